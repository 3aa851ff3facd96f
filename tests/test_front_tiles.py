"""The one-launch front of the build at the sizes where its tiles end, change
their length or find their output offsets in another way."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np

SMALL, LARGE = 2048, 4096  # keys of a tile
DIRECT, SHORT = 96, 152    # tiles up to which counts are added up directly / tiles are short


@pytest.mark.gpu
@pytest.mark.parametrize("n", [LARGE + 1, 3 * SMALL, 3 * SMALL + 1, DIRECT * SMALL, DIRECT * SMALL + 1, SHORT * SMALL,
                               SHORT * SMALL + 1, DIRECT * LARGE, DIRECT * LARGE + 1])
@pytest.mark.parametrize("kind", ["shared", "soup"])
def test_front_at_tile_edges(cuda, oracle, n, kind):
    torch = cuda
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    rng = np.random.default_rng(n)
    if kind == "shared":
        vtx = rng.uniform(-1.0, 1.0, (n // 2 + 3, 3)).astype(np.float32)
        tri = (np.arange(n)[:, None] // 2 + np.array([0, 1, 2])).astype(np.uint32)
    else:  # few distinct codes, and each triangle its own vertices
        vtx = (rng.integers(0, 6, (n, 1, 3)) * 0.125 + rng.integers(0, 2, (n, 3, 3)) * 0.0625).astype(np.float32)
        vtx = vtx.reshape(-1, 3)
        tri = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    ref = oracle.build(tri, vtx)
    for _ in range(2):
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(to_dev(tri, torch), to_dev(vtx, torch))
        assert np.array_equal(to_np(bvh, torch), ref["bvhnodes"])
        assert np.array_equal(bits(to_np(aabb, torch)), bits(ref["bvhnode2aabb"]))
