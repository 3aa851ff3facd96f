"""That the cast's later tiers are reached where they are meant to be, by the cast's own
counters (see cast_job): teams of one warp, a split tier with more rays than its pool
holds, and rays that the split tier hands to the team tier."""
import numpy as np
import pytest

from helpers import bits
from test_tail_tiers import _cast
from test_team_tier import _runs_soup

RAYS, TEAM_RAYS, SPLIT_TO_TEAM, TEAM_TAKES, PARKED = 0, 1, 2, 4, 5  # counters


def _thicket(n, width, seed):
    """Slivers across the unit cube: a ray enters the boxes of hundreds and hits few."""
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(n, 3))
    a *= 0.15 / np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n, 3)))
    b *= width / np.linalg.norm(b, axis=1, keepdims=True)
    c = rng.uniform(0.15, 0.85, (n, 3))
    vtx = np.stack([c - a, c + a - b, c + a + b], 1).reshape(-1, 3).astype(np.float32)
    return np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), vtx


def _aimed(tri, vtx, num_ray, spread, seed):
    from del_msh_gb300 import workloads as W
    rng = np.random.default_rng(seed)
    org, _ = W.cube_boundary_rays(num_ray, seed=seed)
    at = vtx[tri[rng.integers(0, tri.shape[0], num_ray)]].mean(axis=1) + rng.uniform(-spread, spread, (num_ray, 3))
    return org, (at - org).astype(np.float32)


def _check(torch, oracle, tri, vtx, org, d, **tuning):
    from del_msh_gb300 import _native
    ref = oracle.build(tri, vtx)
    r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"])
    assert 0 < (r_hit != 0xFFFFFFFF).sum()
    hit, t, c = _cast(torch, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], org, d, **tuning)
    assert np.array_equal(hit, r_hit)
    assert np.array_equal(bits(t), bits(r_t))
    assert _native.device_status(clear=True) == 0
    return c.astype(np.int64)


@pytest.mark.gpu
def test_teams_of_blocks_and_of_single_warps(cuda, oracle):
    tri, vtx = _runs_soup(3)
    ends = {}
    for num_ray in (3000, 60_000):
        org, d = _aimed(tri, vtx, num_ray, 2e-4, 5)
        c = _check(cuda, oracle, tri, vtx, org, d, cast_long_steps=1)
        assert c[TEAM_RAYS] > 0
        ends[num_ray] = c[TEAM_TAKES] - c[TEAM_RAYS]  # each team takes once too often
    assert ends[60_000] == 4 * ends[3000]  # four warps a block


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2e-4, 2e-3])
def test_more_parked_rays_than_the_pool_holds(cuda, oracle, width):
    from del_msh_gb300 import _native
    tri, vtx = _thicket(20_000, width, 1)
    org, d = _aimed(tri, vtx, 140_001, 0.05, 2)
    c = _check(cuda, oracle, tri, vtx, org, d)
    # half of 64 MiB, and two words of 16 bytes beside each ray's stack
    assert c[PARKED] > (32 << 20) // (16 * (_native.get_tuning()["cast_stack"] + 2))


@pytest.mark.gpu
@pytest.mark.parametrize("num_ray,long_steps", [(3, 30), (3000, 64), (40_000, 140)])
def test_parked_rays_at_long_chains(cuda, oracle, num_ray, long_steps):
    """Past long_steps, which lies beyond the entries at which rays are parked."""
    tri0, vtx0 = _runs_soup(4)
    tri1, vtx1 = _thicket(20_000, 2e-4, 3)
    tri, vtx = np.concatenate([tri0, tri1 + vtx0.shape[0]]).astype(np.uint32), np.concatenate([vtx0, vtx1])
    org, d = _aimed(tri0, vtx0, num_ray, 2e-4, num_ray)
    c = _check(cuda, oracle, tri, vtx, org, d, cast_long_steps=long_steps)
    assert c[PARKED] > 0
    assert c[SPLIT_TO_TEAM] > 0
