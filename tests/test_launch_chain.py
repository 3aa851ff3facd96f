"""Build, refit and cast as one chain of launches over scratch that holds
anything: what each kernel needs zeroed is zeroed by the one before it."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _mesh(n, seed):
    rng = np.random.default_rng(seed)
    m = max(3, int(np.sqrt(n / 2)))
    # n triangles between neighbouring points of a curve: shared vertices
    vtx = np.cumsum(rng.normal(0.0, 1.0, (n // 2 + 3, 3)), axis=0).astype(np.float32) / m
    tri = (np.arange(n)[:, None] // 2 + np.array([0, 1, 2])).astype(np.uint32)
    return tri, vtx


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 257, 4097, 5120, 70001])
@pytest.mark.parametrize("height", [False, True])
def test_dirty_scratch(cuda, oracle, n, height):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _mesh(n, n)
    ref = oracle.build(tri, vtx)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    for fill in (0xFF, 0x5A):
        # the allocator hands the freed block out again as scratch
        size = _native.size("dm_trimesh3_build_scratch_bytes", n)
        dirty = torch.full((size,), fill, dtype=torch.uint8, device="cuda:0")
        del dirty
        out = TriMesh3.make_bvhnodes_bvhnode2aabb_ex(d_tri, d_vtx, want_height=height)
        assert np.array_equal(to_np(out["bvhnodes"], torch), ref["bvhnodes"])
        assert np.array_equal(bits(to_np(out["bvhnode2aabb"], torch)), bits(ref["bvhnode2aabb"]))
        moved = torch.zeros_like(out["bvhnode2aabb"])
        TriMesh3.update_bvhnode2aabb(d_tri, d_vtx, out["bvhnodes"], moved)
        assert np.array_equal(bits(to_np(moved, torch)), bits(ref["bvhnode2aabb"]))
    assert _native.device_status(clear=True) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3000, 5120, 70001])
def test_captured_chain(cuda, oracle, n):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.SearchBvh3 import torch as SearchBvh3
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _mesh(n, n)
    rng = np.random.default_rng(3)
    org = vtx[rng.integers(0, len(vtx), 2000)] + rng.normal(0.0, 0.3, (2000, 3)).astype(np.float32)
    direc = rng.normal(0.0, 1.0, (2000, 3)).astype(np.float32)
    d_tri, d_vtx, d_org, d_dir = (to_dev(a, torch) for a in (tri, vtx, org, direc))

    def chain():
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
        again = torch.empty_like(aabb)
        TriMesh3.update_bvhnode2aabb(d_tri, d_vtx, bvh, again)
        return (bvh, aabb, again) + tuple(SearchBvh3.first_intersection_ray(d_org, d_dir, d_tri, d_vtx, bvh, again))

    chain()  # one-time attributes are set outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = chain()
    for k in range(3):
        d_vtx.copy_(torch.from_numpy((vtx * np.float32(1.0 + 0.25 * k)).astype(np.float32)))
        g.replay()
        torch.cuda.synchronize()
        want = chain()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
        ref = oracle.build(tri, to_np(d_vtx, torch))
        assert np.array_equal(to_np(got[0], torch), ref["bvhnodes"])
        assert np.array_equal(bits(to_np(got[2], torch)), bits(ref["bvhnode2aabb"]))
    assert _native.device_status(clear=True) == 0
