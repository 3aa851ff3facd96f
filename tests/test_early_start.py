"""Kernels that start while the one before them still runs read what it wrote: two
meshes in turn through the same scratch, so that a value read too early is one of the
other mesh's."""
import numpy as np
import pytest

from helpers import bits, to_dev, to_np


@pytest.mark.gpu
@pytest.mark.parametrize("radix", [8, 10])
@pytest.mark.parametrize("n", [5000, 66_001, 400_003])
def test_separate_kernels_in_turn(cuda, oracle, n, radix):
    torch = cuda
    from del_msh_gb300 import _native
    from del_msh_gb300.TriMesh3 import torch as TriMesh3
    meshes = []
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        cen = rng.random((n, 1, 3))
        vtx = (cen + 0.01 * rng.normal(size=(n, 3, 3))).reshape(-1, 3).astype(np.float32)
        tri = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
        meshes.append((to_dev(tri, torch), to_dev(vtx, torch), oracle.build(tri, vtx)))
    before = _native.get_build_classes()
    wrong = torch.zeros((), dtype=torch.int64, device="cuda:0")
    try:
        _native.set_build_classes([dict(max_tri=0xFFFFFFFF, build_path=1, sort_radix=radix, topo_threads=256)])
        want = [(to_dev(r["bvhnodes"], torch).view(torch.int32),
                 to_dev(bits(r["bvhnode2aabb"]), torch).view(torch.int32)) for _, _, r in meshes]
        for k in range(200):
            tri, vtx, _ = meshes[k % 2]
            bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(tri, vtx)
            wrong += (bvh.view(torch.int32) != want[k % 2][0]).sum() + (aabb.view(torch.int32) != want[k % 2][1]).sum()
    finally:
        _native.set_build_classes(before)
    assert int(wrong) == 0
    assert _native.device_status(clear=True) == 0
