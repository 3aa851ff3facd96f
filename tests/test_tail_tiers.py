"""The kernel that finishes a cast: its tiers at the sizes where they change, and that
each of them has run (by the cast's counters in the caller's scratch)."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _cast(torch, tri, vtx, bvh, aabb, org, d, **tuning):
    """Hits, distances and the cast's counters (see cast_job)."""
    from del_msh_gb300 import _native
    T, n = tri.shape[0], org.shape[0]
    dev = [to_dev(a, torch) for a in (org, d, tri, vtx, bvh, aabb)]
    cs = _native.size("dm_cast_scratch_bytes", n, T)
    scr = torch.empty((cs,), dtype=torch.uint8, device="cuda:0")
    hit = torch.empty((n,), dtype=torch.int32, device="cuda:0")
    t = torch.empty((n,), dtype=torch.float32, device="cuda:0")
    p = [a.data_ptr() for a in dev]
    before = _native.get_tuning()
    try:
        _native.set_tuning(**dict(before, **tuning))
        _native.call("dm_search_bvh3_first_intersection_ray", torch.cuda.current_stream().cuda_stream, n, p[0], p[1],
                     hit.data_ptr(), t.data_ptr(), None, T, p[2], vtx.shape[0], p[3], p[4], p[5], scr.data_ptr(), cs)
        counters = to_np(scr[:256].view(torch.int32), torch).view(np.uint32)
    finally:
        _native.set_tuning(**before)
    return to_np(hit, torch).view(np.uint32), to_np(t, torch), counters


def _row_in_one_cell(n):
    """n small triangles in a row in one Morton cell (of an extent that a far triangle
    sets): their tree is a chain, in which a ray through one misses all links' boxes
    beyond it."""
    x = (np.arange(n) + 0.5) / n
    w = 0.4 / n
    zero = np.zeros(n)
    row = np.stack([np.stack([x - w, zero - 1e-3, zero], -1), np.stack([x + w, zero - 1e-3, zero], -1),
                    np.stack([x, zero + 2e-3, zero], -1)], 1)
    far = np.array([[[1100.0, 1100.0, 1100.0], [1101.0, 1100.0, 1100.0], [1100.0, 1101.0, 1100.0]]])
    vtx = np.concatenate([row, far]).reshape(-1, 3).astype(np.float32)
    return np.arange(vtx.shape[0], dtype=np.uint32).reshape(-1, 3), vtx


@pytest.mark.gpu
@pytest.mark.parametrize("repeat", [1, 60])  # by whole blocks, and by single warps
@pytest.mark.parametrize("n", [31, 64, 65, 257, 1000])
def test_chain_left_at_every_link(cuda, oracle, n, repeat):
    """A warp's part of a round is tested 32 links at a time, and the links of one
    group may replace those of the group before."""
    tri, vtx = _row_in_one_cell(n)
    ref = oracle.build(tri, vtx)
    cen = vtx[tri[:n]].mean(axis=1)
    org = np.repeat(cen + np.float32([0, 0, -1]), repeat, axis=0).astype(np.float32)
    d = np.tile(np.float32([0, 0, 1]), (n * repeat, 1))
    hit, t, c = _cast(cuda, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], org, d, cast_long_steps=1)
    assert c[1] > 0  # rays of the team tier
    r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"])
    assert np.array_equal(r_hit, np.repeat(np.arange(n, dtype=np.uint32), repeat))
    assert np.array_equal(hit, r_hit)
    assert np.array_equal(bits(t), bits(r_t))


def _comb(T):
    """A brought tree whose every branch has a leaf on the right and the rest, which is
    nearer to rays that come from below, on the left: a ray through all boxes has a
    frame on each level, and no chain to fold.  The nearer a triangle, the smaller, so
    that rays further out pop frames whose leaves they hit."""
    z = (T - np.arange(T)) / T
    size = 0.2 + np.round(50 * z) / 50
    vtx = np.zeros((T, 3, 3), np.float32)
    vtx[:, :, :2] = size[:, None, None] * np.array([[-2, -2], [4, -2], [-2, 4]])
    vtx[:, :, 2] = z[:, None]
    tri = np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)
    i = np.arange(T - 1)
    bvh = np.full((2 * T - 1, 3), 0xFFFFFFFF, np.uint32)
    bvh[1:T - 1, 0] = i[:-1]
    bvh[:T - 1, 1] = np.where(i < T - 2, i + 1, 2 * T - 2)
    bvh[:T - 1, 2] = T - 1 + i
    bvh[T - 1:, 0] = np.minimum(np.arange(T), T - 2)
    bvh[T - 1:, 1] = np.arange(T)
    aabb = np.empty((2 * T - 1, 6), np.float32)
    aabb[:, :2], aabb[:, 3:5] = -4.0, 8.0  # every ray meets every box
    aabb[T - 1:, 2] = aabb[T - 1:, 5] = z
    aabb[:T - 1, 2], aabb[:T - 1, 5] = z[-1], z[:T - 1]
    org = np.random.default_rng(T).uniform(-1.0, 1.0, (20_000, 3)).astype(np.float32)
    org[:, 2] = -1.0
    return tri, vtx.reshape(-1, 3), bvh, aabb, org, np.tile(np.float32([0, 0, 1]), (20_000, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("T,num_ray", [(60, 3000), (500, 3000), (1300, 3000), (1300, 20_000), (5000, 300),
                                       (30_000, 300), (100_000, 60)])
def test_trees_deeper_than_a_stack(cuda, oracle, T, num_ray):
    """Within the on-chip stack, a team's slice, and with stacks carved from a group's
    share of the pool or (from 14,600 levels on) from the whole."""
    tri, vtx, bvh, aabb, org, d = _comb(T)
    org, d = org[:num_ray], d[:num_ray]
    hit, t, c = _cast(cuda, tri, vtx, bvh, aabb, org, d)
    assert c[5] > 0  # parked
    assert (c[7:32] == 0xFFFFFFFF).all()  # the lists of rays handed on are empty again
    # the last, nearest triangle that holds the ray's point
    near = np.full(num_ray, 0xFFFFFFFF, np.uint32)
    for k in range(T):
        s = vtx[3 * k + 1, 0] / 4
        near[(org[:, 0] > -2 * s) & (org[:, 1] > -2 * s) & (org[:, 0] + org[:, 1] < 2 * s)] = k
    assert np.array_equal(hit, near)
    if T <= 5000:
        r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, bvh, aabb)
        assert np.array_equal(hit, r_hit)
        assert np.array_equal(bits(t), bits(r_t))
