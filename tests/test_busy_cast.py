"""The cast of a server with requests in flight, which parks no rays: long rays and
long chains of equal codes, against the oracle."""
import numpy as np
import pytest

from test_split_tier import _crumpled
from test_team_tier import _runs_soup


@pytest.mark.gpu
@pytest.mark.parametrize("long_steps", [None, 1])
@pytest.mark.parametrize("num_ray", [1, 33, 5000])
def test_requests_in_flight(cuda, oracle, long_steps, num_ray):
    from del_msh_gb300 import _native
    from del_msh_gb300 import workloads as W
    from del_msh_gb300.serve import CAST_RAYS, Request, Server
    meshes = [_crumpled(30, 1), _runs_soup(3)]
    rng = np.random.default_rng(num_ray)
    keep, reqs, expect = [], [], []
    for k in range(16):
        mesh = k % 2
        tri, vtx = meshes[mesh]
        lo, hi = vtx.min(0), vtx.max(0)
        org, _ = W.cube_boundary_rays(num_ray, seed=k + 1)
        org = np.ascontiguousarray(lo + org * (hi - lo), np.float32)
        target = vtx[tri[rng.integers(0, tri.shape[0], num_ray)]].mean(axis=1)
        d = np.ascontiguousarray(target + rng.uniform(-2e-4, 2e-4, (num_ray, 3)) - org, np.float32)
        hit, t = np.zeros(num_ray, np.uint32), np.zeros(num_ray, np.float32)
        keep.append((org, d, hit, t))
        reqs.append(Request(kind=CAST_RAYS, mesh_id=mesh, frame=0, num_ray=num_ray, ray_org=org.ctypes.data,
                            ray_dir=d.ctypes.data, out_tri=hit.ctypes.data, out_t=t.ctypes.data))
        ref = oracle.build(tri, vtx)
        expect.append(oracle.cast_rays(org, d, tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"]))
    before = _native.get_tuning()
    try:
        if long_steps is not None:
            _native.set_tuning(**dict(before, cast_long_steps=long_steps))
        with Server(budget_bytes=4 << 30, num_slots=4, max_tri=max(m[0].shape[0] for m in meshes),
                    max_out=num_ray) as srv:
            for k, (tri, vtx) in enumerate(meshes):
                srv.register(k, tri, vtx, seed=k)
            res = srv.run_trace(reqs, [0.0] * len(reqs))
    finally:
        _native.set_tuning(**before)
    assert all(r.status == 0 for r in res)
    for (_, _, hit, t), (r_hit, r_t) in zip(keep, expect):
        assert np.array_equal(hit, r_hit)
        assert np.array_equal(t.view(np.uint32), r_t.view(np.uint32))
    assert _native.device_status(clear=True) == 0
