"""The cast's team tier: chains of every length at the edges of its rounds, by
whole blocks (few rays) and by single warps (many)."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np

RUNS = [2, 8, 9, 10, 31, 33, 127, 129, 130, 256, 258, 511, 513, 514, 1025, 2050, 5000]


def _runs_soup(seed):
    """Small triangles in runs of equal Morton codes: run k lies inside one cell
    of the 1024^3 grid over the soup, so that its tree is a chain of its length."""
    rng = np.random.default_rng(seed)
    cell = 1.0 / 1024
    cog = [np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]])]  # the soup's extent
    for k, n in enumerate(RUNS):
        at = (np.array([60 * k + 7, 1023 - 55 * k, 31 + 50 * k]) + 0.1) * cell
        cog.append(at + 0.8 * cell * rng.random((n, 3)))
    cog = np.concatenate(cog)
    vtx = cog[:, None, :] + 3e-4 * (rng.random((cog.shape[0], 3, 3)) - 0.5)
    vtx -= vtx.mean(axis=1, keepdims=True) - cog[:, None, :]
    tri = np.arange(3 * cog.shape[0], dtype=np.uint32).reshape(-1, 3)
    order = rng.permutation(cog.shape[0])
    return tri[order], vtx.reshape(-1, 3).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("num_ray,many", [(3000, False), (20000, True)])
def test_chains_of_all_lengths(cuda, oracle, num_ray, many):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300 import workloads as W
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _runs_soup(3)
    rng = np.random.default_rng(num_ray)
    org, _ = W.cube_boundary_rays(num_ray, seed=5)
    target = vtx[tri[rng.integers(0, tri.shape[0], num_ray)]].mean(axis=1) + rng.uniform(-2e-4, 2e-4, (num_ray, 3))
    d = (target - org).astype(np.float32)
    ref = oracle.build(tri, vtx)
    links = ref["bvhnodes"][: tri.shape[0] - 1]
    j = np.arange(tri.shape[0] - 1)
    assert ((links[:, 1] == tri.shape[0] - 1 + j) & (links[:, 2] == j + 1)).sum() > sum(RUNS) - 3 * len(RUNS)
    r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"])
    assert (r_hit != 0xFFFFFFFF).sum() > num_ray // 4
    L = _native.load()
    before = _native.get_tuning()
    d_tri, d_vtx, d_org, d_dir = (to_dev(a, torch) for a in (tri, vtx, org, d))
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    T = tri.shape[0]
    cs = L.dm_cast_scratch_bytes(num_ray, T)
    scr = torch.empty((cs,), dtype=torch.uint8, device="cuda:0")
    hit = torch.empty((num_ray,), dtype=torch.int32, device="cuda:0")
    t = torch.empty((num_ray,), dtype=torch.float32, device="cuda:0")
    try:
        _native.set_tuning(**dict(before, cast_long_steps=1))
        _native.call("dm_search_bvh3_first_intersection_ray", torch.cuda.current_stream().cuda_stream, num_ray,
                     d_org.data_ptr(), d_dir.data_ptr(), hit.data_ptr(), t.data_ptr(), None, T, d_tri.data_ptr(),
                     vtx.shape[0], d_vtx.data_ptr(), bvh.data_ptr(), aabb.data_ptr(), scr.data_ptr(), cs)
        handed = int(scr[4:8].view(torch.int32).item())
    finally:
        _native.set_tuning(**before)
    # up to 8 rays for each of the 608 blocks are cast by whole blocks
    assert handed > 8 * 608 if many else 0 < handed <= 8 * 608
    assert np.array_equal(to_np(hit, torch).view(np.uint32), r_hit)
    assert np.array_equal(bits(to_np(t, torch)), bits(r_t))
    assert _native.device_status(clear=True) == 0
