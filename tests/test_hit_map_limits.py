"""Hit maps with triangles out of range: such a pixel raises the status and is nothing,
whether its output was filled before or is defined by the kernel."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np

BAD_INDEX = 4


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (33, 17), (700, 500)])
def test_triangles_out_of_range(cuda, oracle, w, h):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300 import workloads as W
    from del_msh_gb300.Pix2Depth import torch as Pix2Depth
    from del_msh_gb300.Pix2Tri import torch as Pix2Tri
    tri, vtx = W.displaced_torus(24, seed=4)
    m = W.pinhole_ndc2world(W.random_viewpoint(3.0, seed=3), aspect=w / h)
    row = torch.from_numpy(np.ascontiguousarray(m.reshape(4, 4).T)).to("cuda:0")
    ref = oracle.build(tri, vtx)
    good, _ = oracle.pix2tri(tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], m, w, h)
    good = good.reshape(h, w)
    bad = np.zeros((h, w), bool)
    bad.reshape(-1)[::3] = True
    worse = np.where(bad, np.where(np.arange(w * h).reshape(h, w) % 2 == 0, tri.shape[0], 0xFFFFFFFE), good)
    # the same map with background in their place
    none = to_dev(np.where(bad, 0xFFFFFFFF, good).astype(np.uint32), torch)
    hits = to_dev(worse.astype(np.uint32), torch)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    val = torch.rand((vtx.shape[0], 3), device="cuda:0")
    assert _native.device_status(clear=True) == 0

    def outputs(p2t):
        v, x = d_vtx.clone().requires_grad_(True), val.clone().requires_grad_(True)
        junk = [torch.full((h, w, k), 7.0, device="cuda:0") for k in (1, 3)]  # memory that outputs may get
        del junk
        depth = Pix2Depth.AutogradFunction.apply(v, p2t, d_tri, row)
        pix = Pix2Tri.interpolate(p2t, d_tri, v, x, row)
        (depth.sum() + pix.sum()).backward()
        return depth.detach(), pix.detach(), v.grad, x.grad

    want = outputs(none)
    assert _native.device_status(clear=True) == 0
    got = outputs(hits)
    assert _native.device_status(clear=True) == BAD_INDEX
    assert not to_np(got[0], torch)[bad].any() and not to_np(got[1], torch)[bad].any()
    for a, b in zip(got[:2], want[:2]):
        assert np.array_equal(bits(to_np(a, torch)), bits(to_np(b, torch)))
    # sums of the same terms, up to some thousand a vertex, in another order each
    for a, b in zip(got[2:], want[2:]):
        assert float((a - b).abs().max()) <= 1e-4 * (float(b.abs().max()) + 1e-30)
    # what the caller filled stays
    out = torch.full((h, w), 7.0, device="cuda:0")
    Pix2Depth.update(out, hits, d_tri, d_vtx, row)
    assert _native.device_status(clear=True) == BAD_INDEX
    assert (to_np(out, torch)[bad] == 7.0).all()
