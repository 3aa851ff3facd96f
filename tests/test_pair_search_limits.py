"""The pair search where its lists and stacks run full: no pair may be lost."""
import numpy as np
import pytest

from helpers import to_dev, to_np


def _all_boxes_overlap(nx, ny, nz):
    """Large triangles around the points of a grid, in planes x + y + z = c, and
    one in 64 in a plane x - y = c.  Every box overlaps every other; the tree over
    the grid is balanced.  A triangle of the one kind crosses every triangle of the
    other in the middle, two of a kind lie in parallel planes (all of it exact in
    f32), so the number of pairs is the product of the kinds' numbers."""
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    kind = (g @ np.array([1, 7, 13])) % 64 == 0
    a = 4096.0 * np.array([[2, -1, -1], [-1, 2, -1], [-1, -1, 2]])
    b = 4096.0 * np.array([[1, 1, -1], [-1, -1, -1], [0, 0, 2]])
    vtx = (g[:, None, :] + np.where(kind[:, None, None], b, a)).reshape(-1, 3).astype(np.float32)
    tri = np.arange(vtx.shape[0], dtype=np.uint32).reshape(-1, 3)
    return tri, vtx, int(kind.sum()) * int((~kind).sum())


@pytest.mark.parametrize("grid", [(4, 4, 2), (8, 8, 16)])
def test_all_boxes_overlap_on_the_oracle(oracle, grid):
    tri, vtx, expect = _all_boxes_overlap(*grid)
    r = oracle.build(tri, vtx)
    p, _ = oracle.self_intersection(tri, vtx, r["bvhnodes"], r["bvhnode2aabb"])
    assert len(p) == expect


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(16, 16, 16), (64, 64, 16), (64, 64, 32)])
def test_full_lists_lose_no_pairs(cuda, grid):
    """From 65,536 triangles on the next round's list of 1,048,576 pairs fills up
    while the warps still hold most of the work."""
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx, expect = _all_boxes_overlap(*grid)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    count = torch.empty((1,), dtype=torch.int32, device="cuda:0")
    _native.call("dm_trimesh3_self_intersection", torch.cuda.current_stream().cuda_stream, tri.shape[0],
                 d_tri.data_ptr(), vtx.shape[0], d_vtx.data_ptr(), bvh.data_ptr(), aabb.data_ptr(), 0, None, None,
                 count.data_ptr())
    assert int(to_np(count, torch).view(np.uint32)[0]) == expect
    assert _native.device_status(clear=True) == 0
