"""Argsort above the size where the match-ranked radix pass takes over: at and
around whole tiles, with keys that fill one digit, few digits or all; and the
batched build's sort around whole 32-key slots, with runs of equal codes."""
import numpy as np
import pytest

TILE = 4096
FIRST = 1 << 20  # above the limit of the 10-bit passes


@pytest.mark.gpu
@pytest.mark.parametrize("n", [FIRST + 1, FIRST + TILE - 1, FIRST + TILE, FIRST + TILE + 33, 3 * FIRST + 7])
@pytest.mark.parametrize("keys", ["all", "few", "warp"])
def test_argsort_at_tile_edges(cuda, n, keys):
    import torch
    from del_msh_gb300.Array1D import torch as Array1D

    rng = np.random.default_rng(n)
    k = {
        "all": lambda: rng.integers(0, 1 << 32, n, dtype=np.uint32),
        "few": lambda: rng.integers(0, 3, n, dtype=np.uint32) * np.uint32(0x40404040),
        # runs of 256 equal keys that start anywhere: one digit fills a warp's rank byte
        "warp": lambda: np.repeat(rng.integers(0, 1 << 32, n // 256 + 2, dtype=np.uint32), 256)[77:77 + n],
    }[keys]()
    idx, srt = Array1D.argsort(torch.from_numpy(k.view(np.int32).copy()).view(torch.uint32).cuda())
    ref = np.argsort(k, kind="stable")
    assert np.array_equal(idx.cpu().view(torch.int32).numpy().view(np.uint32), ref.astype(np.uint32))
    assert np.array_equal(srt.cpu().view(torch.int32).numpy().view(np.uint32), k[ref])


@pytest.mark.gpu
def test_batch_sort_at_slot_edges(cuda, oracle):
    import torch
    from del_msh_gb300.batch import MeshBatch

    rng = np.random.default_rng(5)
    meshes = []
    for n in (2, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 2049, 16383):
        # vertices on a coarse grid: many equal centroids, so equal codes
        vtx = (rng.integers(0, 5, (max(n // 2, 3), 3)) * 0.25).astype(np.float32)
        meshes.append((rng.integers(0, len(vtx), (n, 3)).astype(np.uint32), vtx))
    b = MeshBatch(meshes)
    b.build()
    torch.cuda.synchronize()
    for m, (tri, vtx) in enumerate(meshes):
        ref = oracle.build(tri, vtx)
        bvh, aabb = b.mesh_tree(m)
        assert np.array_equal(bvh.cpu().view(torch.int32).numpy().view(np.uint32), ref["bvhnodes"]), m
        assert np.array_equal(aabb.cpu().numpy().view(np.uint32), ref["bvhnode2aabb"].view(np.uint32)), m
