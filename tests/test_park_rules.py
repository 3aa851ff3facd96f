"""Which rays the persistent cast parks: none of a small mesh's ordinary rays, and none
that stands at a long chain, by the cast's own counters (see cast_job)."""
import numpy as np
import pytest

from helpers import bits
from test_tail_tiers import _cast
from test_team_tier import _runs_soup

TEAM_RAYS, PARKED = 1, 5


def _check(torch, oracle, tri, vtx, org, d, **tuning):
    ref = oracle.build(tri, vtx)
    r_hit, r_t = oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"])
    hit, t, c = _cast(torch, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], org, d, **tuning)
    assert np.array_equal(hit, r_hit)
    assert np.array_equal(bits(t), bits(r_t))
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("level,num_ray", [(1, 1), (1, 20_000), (2, 1000), (2, 20_000)])
def test_small_meshes(cuda, oracle, level, num_ray):
    from del_msh_gb300 import workloads as W
    tri, vtx = W.jittered_icosphere(level, seed=0)
    org, d = W.cube_boundary_rays(num_ray, seed=num_ray, lo=-1.0, hi=1.0)
    assert _check(cuda, oracle, tri, vtx, org, d)[PARKED] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("num_ray", [300, 20_000])
def test_rays_at_long_chains(cuda, oracle, num_ray):
    """With no bound of its own on the team tier's rays, the bound on parking is it."""
    from del_msh_gb300 import workloads as W
    tri, vtx = _runs_soup(5)
    rng = np.random.default_rng(num_ray)
    org, _ = W.cube_boundary_rays(num_ray, seed=6)
    at = vtx[tri[rng.integers(0, tri.shape[0], num_ray)]].mean(axis=1) + rng.uniform(-2e-4, 2e-4, (num_ray, 3))
    assert _check(cuda, oracle, tri, vtx, org, (at - org).astype(np.float32), cast_long_steps=1 << 20)[TEAM_RAYS] > 0
