"""Per-pixel closest-hit triangle by BVH ray casting on CUDA tensors.

Mirrors ``del_msh_dlpack/Pix2Tri/torch.py:8-61`` (by_raycasting).  Pixel
(iw, ih) casts the ray of ray_for_pixel.h through ``transform_ndc2world``
(row-major 4x4, read as such: the reference transposes it for its kernel); hits follow del-msh-cpu's search_bvh3::first_intersection_ray.
"""
from __future__ import annotations

from typing import Tuple

import torch

from .. import _native
from .._native import DEFINE_OUTPUT, MATRIX_ROW_MAJOR
from ..util_torch import assert_shape_dtype_device, plain, ptr, require_cuda, scratch, stream_ptr


def by_raycasting(tri2vtx: torch.Tensor, vtx2xyz: torch.Tensor, bvhnodes: torch.Tensor, bvhnode2aabb: torch.Tensor,
                  transform_ndc2world: torch.Tensor, img_shape: Tuple[int, int], return_depth: bool = False):
    """Returns pix2tri (img_h, img_w) uint32 (u32::MAX where nothing is hit);
    with return_depth also pix2t (img_h, img_w) float32, the ray coefficient of
    the hit (+inf on a miss)."""
    num_tri, num_vtx, num_bvhnode = tri2vtx.shape[0], vtx2xyz.shape[0], bvhnodes.shape[0]
    device = tri2vtx.device
    assert num_bvhnode == num_tri * 2 - 1
    assert_shape_dtype_device(tri2vtx, (num_tri, 3), torch.uint32, device)
    assert_shape_dtype_device(vtx2xyz, (num_vtx, 3), torch.float32, device)
    assert_shape_dtype_device(bvhnodes, (num_bvhnode, 3), torch.uint32, device)
    assert_shape_dtype_device(bvhnode2aabb, (num_bvhnode, 6), torch.float32, device)
    assert_shape_dtype_device(transform_ndc2world, (4, 4), torch.float32, device)
    require_cuda(device)
    img_w, img_h = img_shape
    pix2tri = torch.empty((img_h, img_w), dtype=torch.uint32, device=device)
    pix2t = torch.empty((img_h, img_w), dtype=torch.float32, device=device) if return_depth else None
    tri2vtx, vtx2xyz, bvhnodes, bvhnode2aabb, mat = map(
        plain, (tri2vtx, vtx2xyz, bvhnodes, bvhnode2aabb, transform_ndc2world))
    scr = scratch(device, _native.size("dm_cast_scratch_bytes", img_w * img_h, num_tri))
    _native.call("dm_pix2tri_by_raycast_ex", stream_ptr(device), img_w, img_h, ptr(pix2tri), ptr(pix2t), num_tri,
                 ptr(tri2vtx), num_vtx, ptr(vtx2xyz), ptr(bvhnodes), ptr(bvhnode2aabb), ptr(mat), ptr(scr),
                 scr.numel(), MATRIX_ROW_MAJOR)
    return (pix2tri, pix2t) if return_depth else pix2tri


def interpolate_fwd(pix2tri: torch.Tensor, tri2vtx: torch.Tensor, vtx2xyz: torch.Tensor, vtx2val: torch.Tensor,
                    transform_ndc2world: torch.Tensor):
    """pix2val (img_h, img_w, num_vdim): the vertex values interpolated with the
    barycentric coordinates of each pixel's ray on its triangle, 0 on the
    background (``del_msh_dlpack/Pix2Tri/torch.py`` interpolate_fwd)."""
    num_tri, num_vtx, num_vdim = tri2vtx.shape[0], vtx2xyz.shape[0], vtx2val.shape[1]
    img_h, img_w = pix2tri.shape[0], pix2tri.shape[1]
    device = tri2vtx.device
    assert_shape_dtype_device(pix2tri, (img_h, img_w), torch.uint32, device)
    assert_shape_dtype_device(tri2vtx, (num_tri, 3), torch.uint32, device)
    assert_shape_dtype_device(vtx2xyz, (num_vtx, 3), torch.float32, device)
    assert_shape_dtype_device(vtx2val, (num_vtx, num_vdim), torch.float32, device)
    assert_shape_dtype_device(transform_ndc2world, (4, 4), torch.float32, device)
    require_cuda(device)
    pix2tri, tri2vtx, vtx2xyz, vtx2val, mat = map(plain, (pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world))
    pix2val = torch.empty((img_h, img_w, num_vdim), dtype=torch.float32, device=device)  # every pixel is written
    _native.call("dm_pix2tri_interpolate_ex", stream_ptr(device), img_w, img_h, ptr(pix2tri), num_tri, ptr(tri2vtx),
                 num_vtx, ptr(vtx2xyz), num_vdim, ptr(vtx2val), ptr(mat), ptr(pix2val), MATRIX_ROW_MAJOR)
    return pix2val


def interpolate_bwd(pix2tri: torch.Tensor, tri2vtx: torch.Tensor, vtx2xyz: torch.Tensor, vtx2val: torch.Tensor,
                    transform_ndc2world: torch.Tensor, dldw_pix2val: torch.Tensor, dldw_vtx2xyz: torch.Tensor,
                    dldw_vtx2val: torch.Tensor):
    """Adds the backward of interpolate_fwd into dldw_vtx2xyz and dldw_vtx2val."""
    _interpolate_bwd(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world, dldw_pix2val, dldw_vtx2xyz,
                     dldw_vtx2val, 0)


def _interpolate_bwd(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world, dldw_pix2val, dldw_vtx2xyz,
                     dldw_vtx2val, flags):
    num_tri, num_vtx, num_vdim = tri2vtx.shape[0], vtx2xyz.shape[0], vtx2val.shape[1]
    img_h, img_w = pix2tri.shape[0], pix2tri.shape[1]
    device = tri2vtx.device
    assert_shape_dtype_device(pix2tri, (img_h, img_w), torch.uint32, device)
    assert_shape_dtype_device(tri2vtx, (num_tri, 3), torch.uint32, device)
    assert_shape_dtype_device(vtx2xyz, (num_vtx, 3), torch.float32, device)
    assert_shape_dtype_device(vtx2val, (num_vtx, num_vdim), torch.float32, device)
    assert_shape_dtype_device(transform_ndc2world, (4, 4), torch.float32, device)
    assert_shape_dtype_device(dldw_pix2val, (img_h, img_w, num_vdim), torch.float32, device)
    assert_shape_dtype_device(dldw_vtx2xyz, (num_vtx, 3), torch.float32, device)
    assert_shape_dtype_device(dldw_vtx2val, (num_vtx, num_vdim), torch.float32, device)
    require_cuda(device)
    pix2tri, tri2vtx, vtx2xyz, vtx2val, mat, dldw_pix2val = map(
        plain, (pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world, dldw_pix2val))
    _native.call("dm_pix2tri_interpolate_bwd_ex", stream_ptr(device), img_w, img_h, ptr(pix2tri), num_tri,
                 ptr(tri2vtx), num_vtx, ptr(vtx2xyz), num_vdim, ptr(vtx2val), ptr(mat), ptr(dldw_pix2val),
                 ptr(dldw_vtx2xyz), ptr(dldw_vtx2val), MATRIX_ROW_MAJOR | flags)


class AutogradInterpolate(torch.autograd.Function):
    """Differentiable interpolation of vertex values as a torch.autograd.Function."""

    @staticmethod
    def forward(ctx, pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world):
        ctx.save_for_backward(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world)
        return interpolate_fwd(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world)

    @staticmethod
    def backward(ctx, dldw_pix2val):
        pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world = ctx.saved_tensors
        dldw_vtx2xyz = torch.empty(vtx2xyz.shape, dtype=vtx2xyz.dtype, device=vtx2xyz.device)
        dldw_vtx2val = torch.empty(vtx2val.shape, dtype=vtx2val.dtype, device=vtx2val.device)
        _interpolate_bwd(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world, dldw_pix2val, dldw_vtx2xyz,
                         dldw_vtx2val, DEFINE_OUTPUT)
        return None, None, dldw_vtx2xyz, dldw_vtx2val, None


def interpolate(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world):
    return AutogradInterpolate.apply(pix2tri, tri2vtx, vtx2xyz, vtx2val, transform_ndc2world)
