"""Kernels that split one search or one sum over warps and blocks, at the
sizes where the split changes."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _sums(val, idx2onode, onodes):
    """Sums over every ancestor in binary64, and the sums of magnitudes."""
    out = np.zeros((onodes.shape[0], val.shape[1]))
    mag = np.zeros_like(out)
    cur = idx2onode.astype(np.int64)
    v = val.astype(np.float64)
    while cur.size:
        np.add.at(out, cur, v)
        np.add.at(mag, cur, np.abs(v))
        cur = onodes[cur, 0].astype(np.int64)
        keep = cur != 0xFFFFFFFF
        cur, v = cur[keep], v[keep]
    return out, mag


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 31, 33, 1023, 1024, 1025, 40_001])
@pytest.mark.parametrize("vdim,order", [(1, "sorted"), (2, "sorted"), (3, "shuffled"), (4, "sorted"), (4, "shuffled"),
                                        (7, "sorted"), (8, "offset")])
def test_cell_sums(cuda, oracle, n, vdim, order):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.QuadOctTree import torch as QOT
    rng = np.random.default_rng(n + vdim)
    codes = np.sort(rng.choice(1 << 30, n, replace=False)).astype(np.uint32)
    codes[: n // 2] = codes[0] + np.arange(n // 2, dtype=np.uint32)  # half of the points in one small cell
    codes = np.unique(codes)
    n = codes.size
    t = oracle.quad_oct_tree(codes, 3)
    i2o = t["idx2onode"].copy()
    if order == "shuffled":  # leaves in no order: the sums are the same, only combined later
        rng.shuffle(i2o)
    val = (rng.random((n, vdim)) - 0.25).astype(np.float32)
    ref, mag = _sums(val, i2o, t["onodes"])
    d_val = to_dev(val, torch)
    if order == "offset":  # rows of 16 bytes that do not start on 16 bytes
        room = torch.empty((n * vdim + 1,), device="cuda:0")
        room[1:] = d_val.reshape(-1)
        d_val = room[1:].view(n, vdim)
    got = to_np(QOT.aggregate(d_val, to_dev(i2o, torch), to_dev(t["onodes"], torch)), torch)
    # a term passes at most 5 additions per level in its warp, 5 per level in
    # its block and one per block at the node, each of half an ulp of a partial
    # sum no larger than the sum of magnitudes
    adds = 10 * 11 + n // 1024 + 33
    assert (np.abs(got - ref) <= adds * 2.0 ** -24 * mag + 1e-30).all()
    assert _native.device_status(clear=True) == 0


def _grid_pair(n, seed):
    """Two height fields over one square, crossing each other."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.linspace(0, 1, n + 1), np.linspace(0, 1, n + 1), indexing="ij")
    i = np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]
    tri = np.stack([i, i + n + 1, i + n + 2, i, i + n + 2, i + 1], -1).reshape(-1, 3)
    a = np.stack([x, y, 0.03 * rng.standard_normal(x.shape)], -1).reshape(-1, 3)
    b = np.stack([x + 0.3 / n, y + 0.2 / n, 0.03 * rng.standard_normal(x.shape)], -1).reshape(-1, 3)
    return (np.concatenate([tri, tri + a.shape[0]]).astype(np.uint32), np.concatenate([a, b]).astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 5, 17, 120])
@pytest.mark.parametrize("shift", [0, 1])  # boxes on 8 bytes and off them
def test_pairs_of_all_sizes(cuda, oracle, n, shift):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _grid_pair(n, n)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    rp, rs = oracle.self_intersection(tri, vtx, to_np(bvh, torch), to_np(aabb, torch))
    if shift:
        room = torch.empty((aabb.numel() + 1,), device="cuda:0")
        room[1:] = aabb.reshape(-1)
        aabb = room[1:].view(-1, 6)
    segs, pairs = TriMesh3.self_intersection(d_tri, d_vtx, bvh, aabb)
    gp, gs = to_np(pairs, torch), to_np(segs, torch)
    assert len(rp) > 0 or n < 3
    assert len(gp) == len(rp)
    go, ro = np.lexsort((gp[:, 1], gp[:, 0])), np.lexsort((rp[:, 1], rp[:, 0]))
    assert np.array_equal(gp[go], rp[ro])
    assert np.array_equal(bits(gs[go].reshape(-1, 6)), bits(rs[ro].reshape(-1, 6)))
    assert _native.device_status(clear=True) == 0
