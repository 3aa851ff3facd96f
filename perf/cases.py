"""The work this library is used for, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the standing ones,
``draw(rng)`` one more of the same ranges, ``prepare`` the inputs and handles
that a program has in hand, ``run`` one pass through the public entry points,
``work`` the bytes and operations that pass cannot do without, and ``exact``
the computed numbers in 64 bits, from plain torch.

Integer results (trees, codes, hit ids) and boxes are exact: a box is a
selection among the input coordinates, with no rounding.  Results that are
rounded (hit distances, depths, interpolated values, gradients, sums) have a
64-bit value where it is cheap enough to compute.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "del-msh_gb300"))

from del_msh_gb300 import serve, workloads  # noqa: E402
from del_msh_gb300.Array1D import torch as Array1D  # noqa: E402
from del_msh_gb300.batch import MeshBatch  # noqa: E402
from del_msh_gb300.Mortons import torch as Mortons  # noqa: E402
from del_msh_gb300.Pix2Depth import torch as Pix2Depth  # noqa: E402
from del_msh_gb300.Pix2Tri import torch as Pix2Tri  # noqa: E402
from del_msh_gb300.QuadOctTree import torch as QuadOctTree  # noqa: E402
from del_msh_gb300.SearchBvh3 import torch as SearchBvh3  # noqa: E402
from del_msh_gb300.TriMesh3 import torch as TriMesh3  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # one small mesh made and cast once, as an interactive tool or a test does: latency and launches
        dict(name="mesh_1k", op="mesh", shape="ico", n=8, m=0, w=256, h=256, depth=True),
        # an ordinary scanned or modelled mesh in a preview window, ids alone (sizes that no tile divides)
        dict(name="mesh_65k", op="mesh", shape="torus", n=181, m=181, w=641, h=479, depth=False),
        # the headline step: a large mesh built and cast to a full-HD image
        dict(name="mesh_2m_hd", op="mesh", shape="torus", n=1024, m=1024, w=1920, h=1080, depth=True),
        # triangle soup with clustered centroids (runs of equal codes), cast by random rays
        dict(name="soup_4m", op="soup", tri=4194304, rays=1048576),
        # the largest build: a mesh beyond what one cooperative launch holds, tree alone
        dict(name="build_6m", op="mesh", shape="torus", n=1733, m=1733, w=0, h=0, depth=False),
        # a deformed frame of a resident tree: refit, then a 512 x 512 re-cast (the commonest served request)
        dict(name="refit_500k", op="refit", shape="torus", n=499, m=503, w=512, h=512, ccd=False),
        # collision queries on a resident tree: explicit rays with barycentrics
        dict(name="rays_16k", op="rays", shape="ico", n=100, m=0, rays=16384),
        # many small meshes of uneven sizes built and cast at once
        dict(name="batch_1024", op="batch", meshes=1024, lo=64, hi=65536, img=64, sizes=0),
        # particles: codes, sort, oct-tree and the sums over its cells
        dict(name="octree_1m", op="octree", points=1000003, dim=3, vdim=4),
        # differentiable rendering: depth and interpolated colours of a full-HD image, forward and backward
        dict(name="render_hd", op="render", n=1024, m=1024, w=1920, h=1080, vdim=3),
        # cloth and contact: swept boxes for two positions, then the pairs of triangles that cross
        dict(name="contact_260k", op="contact", n=257, m=253),
        # a server's burst: build, refit and ray requests of meshes of different sizes, all outstanding at once
        dict(name="served_mix", op="served", meshes=24, lo=1000, hi=250000, requests=64, img=256, rays=16384, sizes=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi):
    """A torus grid or an icosphere of about a log-uniform number of triangles."""
    t = _log(rng, lo, hi)
    if rng.random() < 0.7 or t > 2000000:
        m = max(3, int(math.sqrt(t / 2) * rng.uniform(0.6, 1.0)))
        return dict(shape="torus", n=max(3, t // (2 * m)), m=m)
    return dict(shape="ico", n=max(1, int(math.sqrt(t / 20))), m=0)


def draw(rng):
    op = rng.choice(["mesh", "mesh", "mesh", "soup", "build", "refit", "rays", "batch", "octree", "render", "contact",
                     "served"])
    if op == "mesh":
        return dict(op="mesh", **_shape(rng, 60, 2000000), w=_log(rng, 32, 1920), h=_log(rng, 32, 1080),
                    depth=rng.random() < 0.5)
    if op == "build":
        return dict(op="mesh", **_shape(rng, 60, 6000000), w=0, h=0, depth=False)
    if op == "soup":
        return dict(op="soup", tri=_log(rng, 50000, 4000000), rays=_log(rng, 10000, 1000000))
    if op == "refit":
        ccd = rng.random() < 0.3
        return dict(op="refit", **_shape(rng, 1000, 2000000), w=0 if ccd else _log(rng, 64, 800),
                    h=0 if ccd else _log(rng, 64, 800), ccd=ccd)
    if op == "rays":
        return dict(op="rays", **_shape(rng, 1000, 1000000), rays=_log(rng, 100, 200000))
    if op == "batch":
        return dict(op="batch", meshes=_log(rng, 16, 1000), lo=64, hi=_log(rng, 1000, 65536), img=rng.choice([17, 32, 64]),
                    sizes=rng.randrange(1, 1000))
    if op == "octree":
        dim = rng.choice([2, 3])
        return dict(op="octree", points=_log(rng, 1000, 1000000), dim=dim, vdim=rng.choice([1, 3, 4]))
    if op == "render":
        n = _log(rng, 16, 1000)
        return dict(op="render", n=n, m=max(3, int(n * rng.uniform(0.5, 1.0))), w=_log(rng, 64, 1920), h=_log(rng, 64, 1080),
                    vdim=rng.choice([1, 3, 4]))
    if op == "contact":
        n = _log(rng, 16, 250)
        return dict(op="contact", n=n, m=max(8, int(n * rng.uniform(0.5, 1.0))))
    return dict(op="served", meshes=_log(rng, 2, 24), lo=1000, hi=_log(rng, 5000, 250000), requests=_log(rng, 4, 64),
                img=_log(rng, 64, 256), rays=_log(rng, 100, 16384), sizes=rng.randrange(1, 1000))


# ------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _u32(a):
    return a.to(torch.int32).contiguous().view(torch.uint32)


def _i32(a):
    """A uint32 result seen as int32 (torch handles few operations on uint32)."""
    return a.view(torch.int32)


@functools.lru_cache(maxsize=8)
def _sphere(freq):
    return workloads.geodesic_sphere(freq)


def _torus(n, m, gen):
    """An n x m grid torus (R = 1, r = 0.3) displaced along the tube normal by
    seeded sinusoids, as workloads.displaced_torus, made on the GPU."""
    i = torch.arange(n, device=DEV)[:, None]
    j = torch.arange(m, device=DEV)[None, :]
    i1, j1 = (i + 1) % n, (j + 1) % m
    v00, v11, v10, v01 = (i * m + j), (i1 * m + j1), (i1 * m + j), (i * m + j1)
    tri = torch.stack([v00, v11, v10, v00, v01, v11], -1).reshape(-1, 3)
    a = i.double() * (2 * math.pi / n)
    b = j.double() * (2 * math.pi / m)
    top = max(2, min(64, n // 8, m // 8))
    f = torch.randint(1, top + 1, (2, 8), generator=gen, device=DEV).tolist()
    ph, wt = (torch.rand((2, 8), generator=gen, device=DEV, dtype=torch.float64)).tolist()
    d = torch.zeros((n, m), device=DEV, dtype=torch.float64)
    for k in range(8):
        d += (0.5 + wt[k] / 2) * torch.sin(f[0][k] * a + f[1][k] * b + 2 * math.pi * ph[k])
    d *= 0.02 / sum(0.5 + x / 2 for x in wt)
    r = 0.3 + d
    r0 = 1.0 + r * torch.cos(b)
    xyz = torch.stack([r0 * torch.sin(a), r0 * torch.cos(a), r * torch.sin(b)], -1)
    return _u32(tri), xyz.reshape(-1, 3).float().contiguous()


def _mesh(case, gen):
    if case["shape"] == "torus":
        return _torus(case["n"], case["m"], gen)
    tri, vtx = _sphere(case["n"])
    vtx = torch.from_numpy(vtx).to(DEV)
    vtx = vtx + 0.02 * (torch.rand(vtx.shape, generator=gen, device=DEV) - 0.5)  # each coordinate +-0.01
    return _u32(torch.from_numpy(tri.astype(np.int32)).to(DEV)), vtx


def _row_major(colmajor):
    return torch.from_numpy(np.ascontiguousarray(colmajor.reshape(4, 4).T)).to(DEV)


def _pinhole(w, h, seed):
    eye = workloads.random_viewpoint(3.0, seed=seed)
    return _row_major(workloads.pinhole_ndc2world(eye, aspect=w / h))


def _camera(case, vtx, seed):
    """Pinhole for the tori, orthographic from above for the spheres."""
    if case["shape"] == "torus":
        return _pinhole(case["w"], case["h"], seed)
    return _row_major(workloads.box_ortho_ndc2world(vtx.amin(0).cpu().numpy(), vtx.amax(0).cpu().numpy()))


def _boundary_rays(n, lo, hi, gen):
    """Rays from random points of a box's faces in random inward directions."""
    face = torch.randint(0, 6, (n,), generator=gen, device=DEV)
    axis, side = face // 2, face % 2
    org = torch.rand((n, 3), generator=gen, device=DEV)
    org.scatter_(1, axis[:, None], side[:, None].float())
    d = torch.randn((n, 3), generator=gen, device=DEV)
    d = d / d.norm(dim=1, keepdim=True)
    along = d.gather(1, axis[:, None])[:, 0] * (1.0 - 2.0 * side.float())
    d = torch.where(along[:, None] < 0, -d, d)
    return (lo + org * (hi - lo)).contiguous(), d.contiguous()


def _facing(case, tri, vtx, cam, p2t):
    """Weights of an image loss: the square of the cosine between a pixel's ray
    and its triangle's normal, so that pixels that graze the surface, whose
    gradients grow without bound, count for little; 0 on the background."""
    ids = _i32(p2t).long().reshape(-1)
    p = vtx[_i32(tri).long()[ids.clamp(min=0)]]
    nrm = torch.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], dim=-1)
    d = _pixel_rays(case, cam)[1].float()
    cos2 = (nrm * d).sum(1) ** 2 / ((nrm * nrm).sum(1) * (d * d).sum(1))
    return torch.where(ids >= 0, cos2, torch.zeros_like(cos2)).reshape(case["h"], case["w"])


def _moved(vtx, gen, amp=0.01):
    """The next frame of a deforming mesh: a smooth seeded displacement."""
    k = 2.0 + 4.0 * torch.rand((3, 3), generator=gen, device=DEV)
    ph = 6.2831853 * torch.rand((3,), generator=gen, device=DEV)
    return (vtx + amp * torch.sin(vtx @ k + ph)).contiguous()


@functools.lru_cache(maxsize=4)
def _ragged(meshes, lo, hi, sizes):
    """Icospheres and tori of uneven sizes; a case's sizes are its own, the
    vertices move with the seed."""
    return workloads.ragged_batch(num_mesh=meshes, tmin=lo, tmax=hi, jitter=0.0, seed=sizes)


def _jittered(meshes, seed):
    rng = np.random.default_rng(seed)
    return [(t, v + rng.uniform(-0.01, 0.01, v.shape).astype(np.float32)) for t, v in meshes]


def _points(case, gen):
    """Points in distinct cells of the code grid, in no order: one per cell, off
    its edges.  The cells are the case's own, so that its trees have one size;
    the points' order and places in their cells come from the seed."""
    n, dim = case["points"], case["dim"]
    side = 1024 if dim == 3 else 65536
    # half uniform, half gathered around a few centres
    own = _gen(n)
    c = torch.rand((8, dim), generator=own, device=DEV, dtype=torch.float64)
    k = 3 * n
    p = torch.rand((k, dim), generator=own, device=DEV, dtype=torch.float64)
    near = c[torch.randint(0, 8, (k,), generator=own, device=DEV)]
    p = torch.where((torch.arange(k, device=DEV) % 2 == 0)[:, None], p, (near + 0.08 * (p - 0.5)).clamp(0.0, 1.0))
    cell = (p * side).long().clamp(0, side - 1)
    key = torch.zeros(k, dtype=torch.int64, device=DEV)
    for d in range(dim):
        key = key * side + cell[:, d]
    key = torch.unique(key)
    if key.numel() < n:
        raise ValueError("too few distinct cells")
    key = key[torch.randperm(key.numel(), generator=own, device=DEV)[:n]]
    key = key[torch.randperm(n, generator=gen, device=DEV)]
    xyz = []
    for d in range(dim):
        xyz.append(key // side ** (dim - 1 - d) % side)
    off = 0.25 + 0.5 * torch.rand((n, dim), generator=gen, device=DEV, dtype=torch.float64)
    return ((torch.stack(xyz, 1) + off) / side).float().contiguous()


class _Burst:
    """A server with its meshes registered, a list of requests and where their answers go."""

    def __init__(self, case, seed):
        meshes = _jittered(_ragged(case["meshes"], case["lo"], case["hi"], case["sizes"]), seed)
        self.out = self.server = None
        n_out = max(case["img"] ** 2, case["rays"])
        self.server = serve.Server(16 << 30, 8, max(t.shape[0] for t, _ in meshes), n_out)
        rng = np.random.default_rng(seed + 1)
        for i, (t, v) in enumerate(meshes):
            self.server.register(i, t, v, seed=int(rng.integers(1 << 30)))
        kinds, which = _requests(case)
        self.out = torch.empty((len(kinds), n_out), dtype=torch.int32).pin_memory()
        self.out_t = torch.empty((len(kinds), n_out), dtype=torch.float32).pin_memory()
        self.out.zero_()
        self.out_t.zero_()
        self.keep, self.reqs = [], []
        for i, (kind, mesh) in enumerate(zip(kinds, which)):
            v = meshes[mesh][1]
            lo, hi = v.min(0), v.max(0)
            r = serve.Request()
            r.kind, r.mesh_id, r.frame, r.deform_amplitude = int(kind), int(mesh), int(rng.integers(0, 50)), 0.01
            if kind == serve.CAST_RAYS:
                o, d = workloads.cube_boundary_rays(case["rays"], seed=int(rng.integers(1 << 30)))
                (a, an), (b, bn) = serve.pinned(o.shape, np.float32), serve.pinned(d.shape, np.float32)
                an[:], bn[:] = lo + o * (hi - lo), d
                self.keep += [a, b]
                r.num_ray, r.ray_org, r.ray_dir = case["rays"], a.data_ptr(), b.data_ptr()
            else:
                cam = np.ascontiguousarray(workloads.box_ortho_ndc2world(lo, hi))
                self.keep.append(cam)
                r.img_w = r.img_h = case["img"]
                r.transform_ndc2world = cam.ctypes.data
            r.out_tri, r.out_t = self.out[i].data_ptr(), self.out_t[i].data_ptr()
            self.reqs.append(r)
        self.arrivals = [0.0] * len(self.reqs)

    def __del__(self):
        if getattr(self, "server", None) is not None:
            self.server.close()


def _requests(case):
    rng = np.random.default_rng(case["sizes"] + 7)
    return rng.choice(3, size=case["requests"], p=(0.2, 0.6, 0.2)), rng.integers(0, case["meshes"], case["requests"])


def prepare(case, seed):
    op, gen = case["op"], _gen(seed)
    if op == "mesh":
        tri, vtx = _mesh(case, gen)
        return dict(case=case, tri=tri, vtx=vtx, cam=_camera(case, vtx, seed) if case["w"] else None)
    if op == "soup":
        n = case["tri"]
        centre = torch.rand((32, 3), generator=gen, device=DEV)
        cog = centre[torch.randint(0, 32, (n,), generator=gen, device=DEV)]
        cog = (cog + 1e-3 * torch.randn((n, 3), generator=gen, device=DEV)).clamp(0.0, 1.0)
        vtx = cog[:, None, :] + 1e-3 * (torch.rand((n, 3, 3), generator=gen, device=DEV) - 0.5)
        org, d = _boundary_rays(case["rays"], 0.0, 1.0, gen)
        return dict(case=case, tri=_u32(torch.arange(3 * n, device=DEV).reshape(-1, 3)),
                    vtx=vtx.reshape(-1, 3).contiguous(), org=org, dir=d)
    if op == "refit":
        tri, vtx = _mesh(case, gen)
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(tri, vtx)
        v0 = _moved(vtx, gen)
        return dict(case=case, tri=tri, vtx=v0, vtx1=_moved(v0, gen) if case["ccd"] else None, bvh=bvh, aabb=aabb,
                    cam=_camera(case, vtx, seed) if case["w"] else None)
    if op == "rays":
        tri, vtx = _mesh(case, gen)
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(tri, vtx)
        org, d = _boundary_rays(case["rays"], vtx.amin(0), vtx.amax(0), gen)
        return dict(case=case, tri=tri, vtx=vtx, bvh=bvh, aabb=aabb, org=org, dir=d)
    if op == "batch":
        meshes = _jittered(_ragged(case["meshes"], case["lo"], case["hi"], case["sizes"]), seed)
        b = MeshBatch(meshes, device=DEV)
        b.alloc_cast(case["img"], case["img"])
        cams = np.stack([workloads.box_ortho_ndc2world(v.min(0), v.max(0)) for _, v in meshes])
        return dict(case=case, batch=b, cams=torch.from_numpy(cams).to(DEV))
    if op == "octree":
        n = case["points"]
        return dict(case=case, pts=_points(case, gen), unit=torch.eye(case["dim"] + 1, device=DEV),
                    val=torch.rand((n, case["vdim"]), generator=gen, device=DEV))
    if op == "render":
        tri, vtx = _torus(case["n"], case["m"], gen)
        cam = _pinhole(case["w"], case["h"], seed)
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(tri, vtx)
        p2t = Pix2Tri.by_raycasting(tri, vtx, bvh, aabb, cam, (case["w"], case["h"]))
        shape = (case["h"], case["w"])
        face = _facing(case, tri, vtx, cam, p2t)
        return dict(case=case, tri=tri, vtx=vtx, cam=cam, p2t=p2t,
                    val=torch.rand((vtx.shape[0], case["vdim"]), generator=gen, device=DEV),
                    g_depth=face * torch.randn(shape, generator=gen, device=DEV),
                    g_val=face[..., None] * torch.randn(shape + (case["vdim"],), generator=gen, device=DEV))
    if op == "contact":
        t, v = _torus(case["n"], case["m"], gen)
        shift = torch.tensor([0.35, 0.2, 0.1], device=DEV)
        vtx = torch.cat([v, v + shift]).contiguous()
        tri = _u32(torch.cat([_i32(t), _i32(t) + v.shape[0]]))
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(tri, vtx)
        room = 16 * (case["n"] + case["m"]) + 1024
        return dict(case=case, tri=tri, vtx=vtx, vtx1=_moved(vtx, gen, 1e-4), bvh=bvh, aabb=aabb,
                    pair=torch.empty((room, 2), dtype=torch.int32, device=DEV),
                    seg=torch.empty((room, 2, 3), device=DEV))
    return dict(case=case, burst=_Burst(case, seed))


# --------------------------------------------------------------------- runs

def run(s):
    case = s["case"]
    op = case["op"]
    if op == "mesh":
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(s["tri"], s["vtx"])
        if not case["w"]:
            return [_i32(bvh), aabb]
        hit = Pix2Tri.by_raycasting(s["tri"], s["vtx"], bvh, aabb, s["cam"], (case["w"], case["h"]),
                                    return_depth=case["depth"])
        return [_i32(bvh), aabb] + ([_i32(hit[0]), hit[1]] if case["depth"] else [_i32(hit)])
    if op == "soup":
        bvh, aabb = TriMesh3.make_bvhnodes_bvhnode2aabb(s["tri"], s["vtx"])
        hit, t = SearchBvh3.first_intersection_ray(s["org"], s["dir"], s["tri"], s["vtx"], bvh, aabb)
        return [_i32(bvh), aabb, _i32(hit), t]
    if op == "refit":
        TriMesh3.update_bvhnode2aabb(s["tri"], s["vtx"], s["bvh"], s["aabb"], s["vtx1"])
        if not case["w"]:
            return [s["aabb"]]
        hit, t = Pix2Tri.by_raycasting(s["tri"], s["vtx"], s["bvh"], s["aabb"], s["cam"], (case["w"], case["h"]),
                                       return_depth=True)
        return [s["aabb"], _i32(hit), t]
    if op == "rays":
        hit, t, bc = SearchBvh3.first_intersection_ray(s["org"], s["dir"], s["tri"], s["vtx"], s["bvh"], s["aabb"],
                                                       return_bc=True)
        return [_i32(hit), t, bc]
    if op == "batch":
        b = s["batch"]
        b.build()
        hit, t = b.cast_pixels(s["cams"])
        return [_i32(b.bvhnodes), b.bvhnode2aabb, _i32(hit), t]
    if op == "octree":
        code = Mortons.make_vtx2morton_from_vtx2co(s["pts"], s["unit"])
        order, code = Array1D.argsort(code)
        tree = QuadOctTree.QuadOctTree()
        tree.construct_from_idx2morton(code, case["dim"])
        total = tree.aggregate(s["val"][_i32(order).long()])
        return [_i32(order), _i32(code), _i32(tree.onodes), _i32(tree.onode2depth), tree.onode2center,
                _i32(tree.idx2onode), tree.idx2center, total]
    if op == "render":
        vtx = s["vtx"].detach().requires_grad_(True)
        val = s["val"].detach().requires_grad_(True)
        depth = Pix2Depth.AutogradFunction.apply(vtx, s["p2t"], s["tri"], s["cam"])
        colour = Pix2Tri.interpolate(s["p2t"], s["tri"], vtx, val, s["cam"])
        g = torch.autograd.grad([depth, colour], [vtx, val], [s["g_depth"], s["g_val"]])
        return [depth.detach(), colour.detach(), g[0], g[1]]
    if op == "contact":
        # boxes swept over the step for the broad phase, then the boxes at its start for the crossings
        swept = torch.empty_like(s["aabb"])
        TriMesh3.update_bvhnode2aabb(s["tri"], s["vtx"], s["bvh"], swept, s["vtx1"])
        seg, pair = TriMesh3.self_intersection(s["tri"], s["vtx"], s["bvh"], s["aabb"])
        pair = _i32(pair)
        # the pairs come in no particular order: a program puts them in one, in its solver's contact buffers
        order = torch.argsort(pair.long()[:, 0] * s["tri"].shape[0] + pair.long()[:, 1])[:s["pair"].shape[0]]
        s["pair"].fill_(-1)
        s["seg"].fill_(0)
        s["pair"][:order.numel()] = pair[order]
        s["seg"][:order.numel()] = seg[order]
        return [swept, s["pair"], s["seg"], pair.shape[0]]
    b = s["burst"]
    b.server.run_trace(b.reqs, b.arrivals)
    return [b.out, b.out_t]


# --------------------------------------------------------------------- work

def _counts(case):
    """Triangles and vertices of a case's mesh."""
    if case.get("shape") == "ico":
        return 20 * case["n"] ** 2, 10 * case["n"] ** 2 + 2
    return 2 * case["n"] * case["m"], case["n"] * case["m"]


def work(case):
    """Inputs read once and outputs written once; a build writes 36 bytes a
    node (2T - 1 of them), a cast 4 or 8 a ray.  Operations: about 60 a
    triangle for a build, 24 for a refit, 400 a ray (some ten boxes and one
    triangle)."""
    op = case["op"]
    if op in ("mesh", "soup"):
        t, v = (case["tri"], 3 * case["tri"]) if op == "soup" else _counts(case)
        r = case["rays"] if op == "soup" else case["w"] * case["h"]
        per = 32 if op == "soup" else 8 if case["depth"] else 4
        return dict(bytes=12 * t + 12 * v + 36 * (2 * t - 1) + per * r, flops=60 * t + 400 * r)
    if op == "refit":
        t, v = _counts(case)
        r = case["w"] * case["h"]
        return dict(bytes=12 * t + (24 if case["ccd"] else 12) * v + 36 * (2 * t - 1) + 8 * r, flops=24 * t + 400 * r)
    if op == "rays":
        # a ray's own bytes, and some ten nodes of 36 bytes and one triangle of 48 for it, at most the whole mesh and tree
        t, v = _counts(case)
        r = case["rays"]
        return dict(bytes=44 * r + min(12 * t + 12 * v + 36 * (2 * t - 1), (2 * 10 * 36 + 48) * r), flops=400 * r)
    if op in ("batch", "served"):
        size = [(t.shape[0], v.shape[0]) for t, v in _ragged(case["meshes"], case["lo"], case["hi"], case["sizes"])]
        if op == "batch":
            t, v, r = sum(a for a, _ in size), sum(b for _, b in size), case["meshes"] * case["img"] ** 2
            return dict(bytes=12 * t + 12 * v + 36 * (2 * t - case["meshes"]) + 8 * r, flops=60 * t + 400 * r)
        total = flops = 0
        for kind, mesh in zip(*_requests(case)):
            t, v = size[mesh]
            r = case["rays"] if kind == serve.CAST_RAYS else case["img"] ** 2
            total += 8 * r + (24 * r if kind == serve.CAST_RAYS else 12 * t + 24 * v + 36 * (2 * t - 1))
            flops += 400 * r + (0 if kind == serve.CAST_RAYS else (60 if kind == serve.BUILD_CAST else 24) * t)
        return dict(bytes=total, flops=flops)
    if op == "octree":
        n, dim, vd = case["points"], case["dim"], case["vdim"]
        nodes = n // 4  # oct-tree nodes above the points, at least about this many
        link = 1 + 2 ** dim
        return dict(bytes=n * (4 * dim + 4 * vd + 4 + 4 + 4 + 4 * dim) + nodes * 4 * (link + 1 + dim + vd),
                    flops=n * (40 + 4 * vd))
    if op == "render":
        n, px, vd = case["n"] * case["m"], case["w"] * case["h"], case["vdim"]
        # both images out, both gradients in, ids read once a direction, gradients of every vertex
        # written; the mesh under the fifth of the pixels that hit
        return dict(bytes=px * (4 + 4 * vd) * 2 + 8 * px + n * (12 + 4 * vd) + min(n, px // 5) * (36 + 4 * vd),
                    flops=px // 5 * (400 + 30 * vd))
    t = 4 * case["n"] * case["m"]
    return dict(bytes=12 * t + 24 * (t // 2) + 36 * (2 * t - 1), flops=60 * t)


# ----------------------------------------------------------- 64-bit results

def _pixel_rays(case, cam):
    m = cam.double()
    x = 2.0 * (torch.arange(case["w"], device=DEV, dtype=torch.float64) + 0.5) / case["w"] - 1.0
    y = 1.0 - 2.0 * (torch.arange(case["h"], device=DEV, dtype=torch.float64) + 0.5) / case["h"]
    y, x = torch.meshgrid(y, x, indexing="ij")
    one = torch.ones_like(x)
    q0 = torch.stack([x, y, one, one], -1).reshape(-1, 4) @ m.T
    q1 = torch.stack([x, y, -one, one], -1).reshape(-1, 4) @ m.T
    q0, q1 = q0[:, :3] / q0[:, 3:], q1[:, :3] / q1[:, 3:]
    return q0, q1 - q0


def _cross_rays(p0, e1, e2, org, d):
    """Moller-Trumbore of rays (r, 1, 3) with triangles (1, t, 3) or pairwise: t, u, v, det."""
    pv = torch.cross(d, e2, dim=-1)
    det = (e1 * pv).sum(-1)
    tv = org - p0
    u = (tv * pv).sum(-1) / det
    qv = torch.cross(tv, e1.expand_as(tv), dim=-1)
    return (e2 * qv).sum(-1) / det, u, (d * qv).sum(-1) / det, det


def _brute_force(tri, vtx, org, d):
    """Closest hit of every ray by testing every triangle: t (inf: none), u, v."""
    p = vtx.double()[_i32(tri).long()]
    p0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    step = max(1, 20000000 // p0.shape[0])
    found = []
    for k in range(0, org.shape[0], step):
        o, dd = org[k:k + step, None].double(), d[k:k + step, None].double()
        shape = (o.shape[0], p0.shape[0], 3)
        t, u, v, det = _cross_rays(p0[None].expand(shape), e1[None].expand(shape), e2[None].expand(shape),
                                   o.expand(shape), dd.expand(shape))
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
        best, at = torch.where(ok, t, math.inf).min(1)
        at = at[:, None]
        found.append((best, u.gather(1, at)[:, 0], v.gather(1, at)[:, 0]))
    return [torch.cat(x) for x in zip(*found)]


def _tree_boxes(tri, bvh, v0, v1):
    """Boxes of a given tree, level by level from the leaves."""
    nodes = _i32(bvh).long()
    num, t = nodes.shape[0], (nodes.shape[0] + 1) // 2
    p = v0.double()[_i32(tri).long()]
    if v1 is not None:
        p = torch.cat([p, v1.double()[_i32(tri).long()]], 1)
    leaf = nodes[t - 1:, 1]
    box = torch.empty((num, 6), dtype=torch.float64, device=DEV)
    box[t - 1:, :3], box[t - 1:, 3:] = p.amin(1)[leaf], p.amax(1)[leaf]
    levels = [torch.zeros(1, dtype=torch.int64, device=DEV)]
    while True:
        below = nodes[levels[-1], 1:].reshape(-1)
        below = below[below < t - 1]
        if not below.numel():
            break
        levels.append(below)
    for at in reversed(levels):
        a, b = box[nodes[at, 1]], box[nodes[at, 2]]
        box[at] = torch.cat([torch.minimum(a[:, :3], b[:, :3]), torch.maximum(a[:, 3:], b[:, 3:])], 1)
    return box


def _spread(x, gap):
    """The bits of x, `gap` apart."""
    out = torch.zeros_like(x)
    for b in range(16):
        out |= ((x >> b) & 1) << (b * gap)
    return out


def _cell_sums(pts, val, dim):
    """The sums of val over the cells of the quad/oct-tree, in 64 bits: nodes in
    the order of the radix-tree branches (a branch is named by the end of its
    range at its parent's split) that begin a new level of cells."""
    side, levels = (1024, 10) if dim == 3 else (65536, 16)
    cell = (pts.double() * side).long()
    code = sum(_spread(cell[:, d], dim) << (dim - 1 - d) for d in range(dim))
    code, order = torch.sort(code)
    n = code.numel()
    if n < 2:
        return None
    run = torch.cat([torch.zeros((1, val.shape[1]), dtype=torch.float64, device=DEV), val.double()[order].cumsum(0)])
    # level of the smallest cell that holds codes i and i + 1
    x = code[1:] ^ code[:-1]
    top = torch.frexp(x.double())[1].long() - 1
    level = levels - 1 - top // dim
    # every cell with more than one child begins where its codes do: one per (prefix, level) of a split pair
    prefix = (code[:-1] >> (dim * (levels - level))) << (dim * (levels - level))
    key = torch.unique(torch.stack([level, prefix], 1), dim=0)
    level, prefix = key[:, 0].contiguous(), key[:, 1].contiguous()
    lo = torch.searchsorted(code, prefix)
    hi = torch.searchsorted(code, prefix + (torch.ones_like(level) << (dim * (levels - level))))
    # the branch that covers the cell is named by its first code if it is a right child, by its last otherwise
    before = torch.where(lo > 0, code[(lo - 1).clamp(min=0)] ^ code[lo], torch.full_like(lo, 1 << 40))
    after = torch.where(hi < n, code[(hi - 1)] ^ code[hi.clamp(max=n - 1)], torch.full_like(lo, 1 << 40))
    name = torch.where(before < after, lo, hi - 1)
    name = torch.where((lo == 0) & (hi == n), torch.zeros_like(lo), name)
    at = torch.argsort(name)
    return (run[hi] - run[lo])[at]


def exact(case, seed):
    op = case["op"]
    if op in ("soup", "batch", "served", "contact"):
        return None
    if op == "mesh":
        t, _ = _counts(case)
        if not case["w"] or not case["depth"] or t * case["w"] * case["h"] > 2e9:
            return None
        s = prepare(case, seed)
        org, d = _pixel_rays(case, s["cam"])
        return [None, None, None, _brute_force(s["tri"], s["vtx"], org, d)[0].reshape(case["h"], case["w"])]
    if op == "rays":
        t, _ = _counts(case)
        if t * case["rays"] > 6e9:
            return None
        s = prepare(case, seed)
        t, u, v = _brute_force(s["tri"], s["vtx"], s["org"], s["dir"])
        bc = torch.stack([1 - u - v, u, v], 1)
        return [None, t, torch.where(torch.isfinite(t)[:, None], bc, torch.zeros_like(bc))]
    s = prepare(case, seed)
    if op == "refit":
        return [_tree_boxes(s["tri"], s["bvh"], s["vtx"], s["vtx1"]), None, None][:1 if not case["w"] else 3]
    if op == "octree":
        return [None] * 7 + [_cell_sums(s["pts"], s["val"], case["dim"])]
    # render: the hit pixels' rays meet their triangles' planes; gradients by autograd
    vtx = s["vtx"].double().requires_grad_(True)
    val = s["val"].double().requires_grad_(True)
    ids = _i32(s["p2t"]).long().reshape(-1)
    at = torch.nonzero(ids >= 0)[:, 0]
    corner = _i32(s["tri"]).long()[ids[at]]
    p = vtx[corner]
    org, d = _pixel_rays(case, s["cam"])
    org, d = org[at], d[at]
    t, u, v, _ = _cross_rays(p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], org, d)
    q = org + t[:, None] * d
    to_ndc = torch.linalg.inv(s["cam"].double())
    ndc = torch.cat([q, torch.ones_like(q[:, :1])], 1) @ to_ndc.T
    px, vd = case["w"] * case["h"], case["vdim"]
    depth = torch.zeros(px, dtype=torch.float64, device=DEV).index_put((at,), (ndc[:, 2] / ndc[:, 3] + 1) / 2)
    c = val[corner]
    colour = (1 - u - v)[:, None] * c[:, 0] + u[:, None] * c[:, 1] + v[:, None] * c[:, 2]
    colour = torch.zeros((px, vd), dtype=torch.float64, device=DEV).index_put((at,), colour)
    depth, colour = depth.reshape(case["h"], case["w"]), colour.reshape(case["h"], case["w"], vd)
    g = torch.autograd.grad([depth, colour], [vtx, val], [s["g_depth"].double(), s["g_val"].double()])
    return [depth.detach(), colour.detach(), g[0], g[1]]
