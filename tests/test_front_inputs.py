"""The torch front-ends on inputs that are not laid out as the kernels want them,
and outputs that are defined by the kernels and not by a fill before them."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _scene(torch, w, h):
    from del_msh_gb300 import workloads as W
    tri, vtx = W.displaced_torus(24, seed=4)
    m = W.pinhole_ndc2world(W.random_viewpoint(3.0, seed=3), aspect=w / h)
    row = torch.from_numpy(np.ascontiguousarray(m.reshape(4, 4).T)).to("cuda:0")
    return tri, vtx, m, row


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (31, 17), (700, 500)])
def test_layouts(cuda, oracle, w, h):
    torch = cuda
    from del_msh_gb300.Pix2Depth import torch as Pix2Depth
    from del_msh_gb300.Pix2Tri import torch as Pix2Tri
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx, m, row = _scene(torch, w, h)
    ref = oracle.build(tri, vtx)
    r_p2t, r_t = oracle.pix2tri(tri, vtx, ref["bvhnodes"], ref["bvhnode2aabb"], m, w, h)
    # every input strided; the copies must not share memory with each other
    wide = lambda a: torch.cat([a.view(torch.int32) if a.dtype == torch.uint32 else a] * 2, 1)[:, :a.shape[1]]
    s_tri = wide(to_dev(tri, torch)).view(torch.uint32)
    s_vtx = wide(to_dev(vtx, torch))
    assert not s_tri.is_contiguous() and not s_vtx.is_contiguous()
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(s_tri, s_vtx)
    assert np.array_equal(to_np(bvh, torch), ref["bvhnodes"])
    for cam in (row, row.T.contiguous().T):  # row-major, and a transposed view
        p2t, t = Pix2Tri.by_raycasting(s_tri, s_vtx, bvh, aabb, cam, (w, h), return_depth=True)
        assert np.array_equal(to_np(p2t, torch), r_p2t)
        assert np.array_equal(bits(to_np(t, torch)), bits(r_t))
    # a hit map whose triangles the pixels' rays mostly miss, and one out of range
    wrong = to_dev(np.where(r_p2t == 0xFFFFFFFF, r_p2t, (r_p2t + 577) % tri.shape[0]).astype(np.uint32), torch)
    for hits in (p2t, wrong):
        out = torch.zeros((h, w), device="cuda:0")
        Pix2Depth.update(out, hits, s_tri, s_vtx, row)
        junk = torch.full((h, w), 7.0, device="cuda:0")  # freed memory that the next output may get
        del junk
        got = Pix2Depth.AutogradFunction.apply(s_vtx, hits, s_tri, row)
        assert np.array_equal(bits(to_np(got, torch)), bits(to_np(out, torch)))
        # gradients: set by the autograd functions, added by the plain entries
        v = s_vtx.detach().clone().requires_grad_(True)
        g = torch.ones((h, w), device="cuda:0")
        (Pix2Depth.AutogradFunction.apply(v, hits, s_tri, row) * g).sum().backward()
        acc = torch.zeros_like(v)
        Pix2Depth.bwd_wrt_vtx2xyz(acc, hits, s_tri, v, g, row)
        Pix2Depth.bwd_wrt_vtx2xyz(acc, hits, s_tri, v, g, row)
        scale = float(acc.abs().max()) + 1e-30
        # two sums of the same terms in another order each
        assert float((acc - 2 * v.grad).abs().max()) <= 1e-5 * scale
