"""Meshes built by one block: every output against the oracle, at the sizes where
keys per thread, the heap and the last block-built mesh change."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


def _soup(n, kind):
    rng = np.random.default_rng(n)
    vtx = rng.random((n + 2, 3)).astype(np.float32)
    if kind == "runs":  # runs of equal codes of many lengths
        vtx = (np.round(vtx * 6) / 6).astype(np.float32) + (1e-5 * rng.random(vtx.shape)).astype(np.float32)
    elif kind == "same":
        vtx[:] = vtx[0]
    elif kind == "zeros":  # extremes that tie between -0 and +0
        vtx[:, 2] = np.where(rng.random(n + 2) < 0.5, np.float32(-0.0), np.float32(0.0))
    elif kind == "nan":
        vtx[n // 3] = np.nan
        vtx[n // 2, 1] = np.nan
    tri = np.stack([np.arange(n), np.arange(n) + 1, np.arange(n) + 2], 1)
    if kind == "runs":
        tri[:] = rng.integers(0, n + 2, (n, 1))  # three times the same vertex: centroids repeat
    return tri.astype(np.uint32), vtx


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "runs", "same", "zeros", "nan"])
@pytest.mark.parametrize("n", [2, 3, 31, 64, 65, 1000, 1024, 1025, 2048, 2049, 4095, 4096, 4097])
def test_small_build(cuda, oracle, n, kind):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    tri, vtx = _soup(n, kind)
    ref = oracle.build(tri, vtx)
    d_tri, d_vtx = to_dev(tri, torch), to_dev(vtx, torch)
    got = TriMesh3.make_bvhnodes_bvhnode2aabb_ex(d_tri, d_vtx, want_height=False)
    for name in ("tri2morton", "idx2tri", "idx2morton", "bvhnodes"):
        assert np.array_equal(to_np(got[name], torch), ref[name]), name
    assert np.array_equal(bits(to_np(got["bvhnode2aabb"], torch)), bits(ref["bvhnode2aabb"]))
    bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(d_tri, d_vtx)
    assert np.array_equal(to_np(bvh, torch), ref["bvhnodes"])
    assert np.array_equal(bits(to_np(aabb, torch)), bits(ref["bvhnode2aabb"]))
    assert _native.device_status(clear=True) == 0
