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


def _one_long_chain(n):
    """A triangle across n small ones in a row, all in one Morton cell (of an
    extent that a far triangle sets): the tree is a chain over them, and only the
    first triangle's box overlaps the rest of it, so that its search goes down the
    whole chain, one link after the other."""
    x = (np.arange(n) + 0.5) / n
    w = 0.4 / n
    zero = np.zeros(n)
    small = np.stack([np.stack([x - w, zero - 1e-3, zero], -1), np.stack([x + w, zero - 1e-3, zero], -1),
                      np.stack([x, zero + 2e-3, zero], -1)], 1)
    across = np.array([[[-0.5, 0.0, -0.5], [1.5, 0.0, -0.5], [0.5, 0.0, 1.5]]])
    far = 1100.0 + across
    vtx = np.concatenate([across, small, far]).reshape(-1, 3).astype(np.float32)
    return np.arange(vtx.shape[0], dtype=np.uint32).reshape(-1, 3), vtx


def test_long_chain_on_the_oracle(oracle):
    tri, vtx = _one_long_chain(3000)
    r = oracle.build(tri, vtx)
    i = np.arange(tri.shape[0] - 1)
    bvh = r["bvhnodes"][: tri.shape[0] - 1]
    assert ((bvh[:, 1] == tri.shape[0] - 1 + i) & (bvh[:, 2] == i + 1)).sum() >= 2998
    p, _ = oracle.self_intersection(tri, vtx, r["bvhnodes"], r["bvhnode2aabb"])
    assert len(p) == 3000 and (np.sort(p, axis=1)[:, 0] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3000, 150_000, 300_000])
def test_long_chain_loses_no_pairs(cuda, n):
    """A round takes a lone search 32 links further, and there were 4000 rounds."""
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _one_long_chain(n)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    _, pairs = TriMesh3.self_intersection(d_tri, d_vtx, bvh, aabb)
    p = np.sort(to_np(pairs, torch), axis=1)
    assert (p[:, 0] == 0).all()
    assert np.array_equal(np.sort(p[:, 1]), np.arange(1, n + 1))
    assert _native.device_status(clear=True) == 0


def _cyclic_chain(T):
    """A brought tree whose last branch leads back to the first: no search of it ends."""
    tri, vtx = _one_long_chain(T - 2)
    i = np.arange(T - 1)
    bvh = np.zeros((2 * T - 1, 3), np.uint32)
    bvh[:, 0] = 0xFFFFFFFF
    bvh[: T - 1, 1] = T - 1 + i
    bvh[: T - 1, 2] = i + 1
    bvh[T - 2, 2] = 1
    bvh[T - 1:, 1] = np.arange(T)
    bvh[T - 1:, 2] = 0xFFFFFFFF
    aabb = np.tile(np.array([0, 0, 0, 1, 1, 1], np.float32), (2 * T - 1, 1))
    return tri, vtx, bvh, aabb


@pytest.mark.gpu
@pytest.mark.parametrize("T", [3, 50, 2000])
def test_search_without_an_end_is_reported(cuda, T):
    torch = cuda
    from del_msh_gb300 import _native
    tri, vtx, bvh, aabb = (to_dev(a, torch) for a in _cyclic_chain(T))
    count = torch.empty((1,), dtype=torch.int32, device="cuda:0")
    _native.device_status(clear=True)
    _native.call("dm_trimesh3_self_intersection", torch.cuda.current_stream().cuda_stream, T, tri.data_ptr(),
                 vtx.shape[0], vtx.data_ptr(), bvh.data_ptr(), aabb.data_ptr(), 0, None, None, count.data_ptr())
    torch.cuda.synchronize()
    assert _native.device_status(clear=True) & 6  # a bad tree, or pairs left when the rounds ran out
