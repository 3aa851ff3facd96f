"""The cast's split tier: long rays parked by the persistent cast and searched
by several lanes, at the sizes where rays per warp, parking and helping change."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _crumpled(n, seed):
    """A sphere whose vertices move by more than their distance: boxes overlap
    heavily and a ray enters hundreds of nodes."""
    from del_msh_gb300 import workloads as W
    tri, vtx = W.geodesic_sphere(n)
    rng = np.random.default_rng(seed)
    return tri, (vtx + rng.uniform(-2.0 / n, 2.0 / n, vtx.shape)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("num_ray", [1, 3, 4865, 30_000, 140_001])
def test_long_rays(cuda, oracle, num_ray):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300 import workloads as W
    from del_msh_gb300.SearchBvh3 import torch as SearchBvh3
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _crumpled(60, 1)
    lo, hi = vtx.min(0), vtx.max(0)
    org, d = W.cube_boundary_rays(num_ray, seed=num_ray)
    org = (lo + org * (hi - lo)).astype(np.float32)
    # every other ray grazes the surface, so that it misses most of what it enters
    rng = np.random.default_rng(num_ray)
    p = rng.normal(size=(num_ray, 3))
    p = p / np.linalg.norm(p, axis=1, keepdims=True) * 1.02
    t = np.cross(p, rng.normal(size=(num_ray, 3)))
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    org[::2], d[::2] = (p - 3.0 * t)[::2].astype(np.float32), t[::2].astype(np.float32)
    ref = oracle.build(tri, vtx)
    r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"])
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    hit, tt = SearchBvh3.first_intersection_ray(to_dev(org, torch), to_dev(d, torch), d_tri, d_vtx, bvh, aabb)
    assert np.array_equal(to_np(hit, torch), r_hit)
    assert np.array_equal(bits(to_np(tt, torch)), bits(r_t))
    assert _native.device_status(clear=True) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("threads,stack", [(64, 64), (128, 32), (128, 96), (256, 64)])
def test_parked_stacks_of_every_variant(cuda, oracle, threads, stack):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300 import workloads as W
    from del_msh_gb300.Pix2Tri import torch as Pix2Tri
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _crumpled(40, 2)
    m = W.box_ortho_ndc2world(vtx.min(0), vtx.max(0))
    ref = oracle.build(tri, vtx)
    r_p2t, r_tt = oracle.pix2tri(tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], m, 131, 77)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    m_row = torch.from_numpy(np.ascontiguousarray(m.reshape(4, 4).T)).to("cuda:0")
    before = _native.get_tuning()
    try:
        _native.set_tuning(**dict(before, cast_threads=threads, cast_stack=stack))
        p2t, tt = Pix2Tri.by_raycasting(d_tri, d_vtx, bvh, aabb, m_row, (131, 77), return_depth=True)
    finally:
        _native.set_tuning(**before)
    assert np.array_equal(to_np(p2t, torch), r_p2t)
    assert np.array_equal(bits(to_np(tt, torch)), bits(r_tt))
    assert _native.device_status(clear=True) == 0


@pytest.mark.gpu
def test_long_rays_of_several_meshes(cuda, oracle):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.batch import MeshBatch, ortho_transforms
    meshes = [_crumpled(n, n) for n in (3, 20, 45, 7, 50)]
    b = MeshBatch(meshes)
    b.alloc_cast(33, 65)
    cams = ortho_transforms(meshes)
    b.build()
    hit, tt = b.cast_pixels(torch.from_numpy(cams).to("cuda:0"))
    for k, (tri, vtx) in enumerate(meshes):
        ref = oracle.build(tri, vtx)
        r_p2t, r_tt = oracle.pix2tri(tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], cams[k], 33, 65)
        assert np.array_equal(to_np(hit[k], torch), r_p2t)
        assert np.array_equal(bits(to_np(tt[k], torch)), bits(r_tt))
    assert _native.device_status(clear=True) == 0
