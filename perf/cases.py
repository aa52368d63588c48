"""The calls whose speed matters to a program that traces with surface_b200.

Each case is one pass through the public entry points over inputs of a stated
size: LBVH builds and closest-hit traces of every primitive kind, the batched
build and trace, a render graph's frame, the volume march with and without its
adjoint, and the texture fetch.  ``listed()`` names the sizes that stand for
each use; ``draw()`` gives others of the same ranges, odd ones among them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from surface_b200 import scenes as S
from surface_b200 import volume as V
from surface_b200.accel import (Mesh, ParticleAccel, Particles, TetraAccel, Tetrahedron,
                                TriangleAccel, spawn_secondary)
from surface_b200.batch import TriangleBatch
from surface_b200.camera import camera_rays, framebuffer_write, make_camera
from surface_b200.lines import LineAccel, Lines
from surface_b200.scene import RenderGraph
from surface_b200.solids import Solid, SolidAccel
from surface_b200.texture import Texture3D

FLT_MAX = float(np.finfo(np.float32).max)
EXACT_PAIRS = 4.0e10  # ray-triangle pairs a double-precision check of every pair may take


def listed():
    return [
        # a small mesh rebuilt and traced every frame (a cursor, a gizmo, a preview
        # tile): launches and latency
        dict(name="tri_small", kind="triangles", faces=2050, width=96, height=64, isect=False),
        # the plain configuration: an animated mesh of 131,072 triangles, rebuilt and
        # seen through a 512 x 512 camera
        dict(name="tri_frame", kind="triangles", faces=131072, width=512, height=512,
             isect=False),
        # a large mesh with an odd face count and a wide image, with the shading
        # records (position, normal, tangent frame) a renderer reads
        dict(name="tri_shade", kind="triangles", faces=1000003, width=1280, height=720,
             isect=True),
        # a simulation's tetrahedral mesh with a scalar at its vertices, cut by an
        # orthographic view
        dict(name="tet_scalar", kind="tetrahedra", cells=64, width=1024, height=1024,
             double=False),
        # a particle simulation's frame: rebuild, primary rays, one bounce per hit
        dict(name="particles", kind="spheres", count=16777216, width=2048, height=2048),
        # many uneven meshes and views built and traced together
        dict(name="batch", kind="batch", scenes=64, faces=1000000, side=1024),
        # fitting a volume and its transfer function to an image: forward, loss, adjoint
        dict(name="volume_fit", kind="volume", res=256, width=512, height=512, backward=True,
             remap=False),
        # viewing a volume on a stretched grid (coordinate table, repeat wrap)
        dict(name="volume_view", kind="volume", res=192, width=640, height=360, backward=False,
             remap=True),
        # a render graph's frame: moved elements, top-level build, eye rays, trace,
        # framebuffer
        dict(name="scene", kind="scene", grid=4, side=1024),
        # hair: capped cylinders, closest hit and normal, accel kept between frames
        dict(name="lines", kind="lines", strands=100000, segments=16, width=1024, height=1024),
        # a finite-element mesh of hexahedra, rebuilt and traced for position and normal
        dict(name="solids", kind="solids", verts=8, cells=64, width=512, height=512),
        # fetches of a sparse paged volume along march rays
        dict(name="texture", kind="texture", pages=16, page=32, width=512, height=512, steps=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["triangles", "triangles", "tetrahedra", "spheres", "batch", "volume",
                       "scene", "lines", "solids", "texture"])
    image = dict(width=_log(rng, 64, 1400), height=_log(rng, 64, 1024))
    if kind == "triangles":
        return dict(kind=kind, faces=_log(rng, 1024, 2000000), isect=rng.random() < 0.4, **image)
    if kind == "tetrahedra":
        return dict(kind=kind, cells=_log(rng, 6, 64), double=rng.random() < 0.3, **image)
    if kind == "spheres":
        return dict(kind=kind, count=_log(rng, 1024, 12000000), **image)
    if kind == "batch":
        return dict(kind=kind, scenes=_log(rng, 2, 64), faces=_log(rng, 4000, 600000),
                    side=rng.choice([256, 512, 1024]))
    if kind == "volume":
        return dict(kind=kind, res=_log(rng, 24, 256), width=_log(rng, 64, 512),
                    height=_log(rng, 64, 512), backward=rng.random() < 0.6,
                    remap=rng.random() < 0.4)
    if kind == "scene":
        return dict(kind=kind, grid=rng.randint(1, 4), side=_log(rng, 128, 1024))
    if kind == "lines":
        return dict(kind=kind, strands=_log(rng, 100, 100000), segments=rng.randint(5, 16),
                    **image)
    if kind == "solids":
        verts = rng.choice([8, 6, 5])
        return dict(kind=kind, verts=verts, cells=_log(rng, 11, {8: 64, 6: 48, 5: 32}[verts]),
                    width=_log(rng, 64, 512), height=_log(rng, 64, 512))
    return dict(kind=kind, pages=rng.randint(3, 16), page=rng.choice([8, 16, 32]),
                width=_log(rng, 64, 512), height=_log(rng, 64, 512), steps=rng.randint(16, 64))


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape, lo=0.0, hi=1.0):
    u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    return lo + (hi - lo) * u


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _sphere_mesh(faces, g, amplitude=0.1):
    """A sphere through the octahedral map of a square grid, displaced radially by
    value noise: (vertices float32 (V, 3), faces int32 (faces, 3))."""
    m = max(2, math.isqrt((faces + 1) // 2))
    while 2 * m * m < faces:
        m += 1
    ax = torch.linspace(-1.0, 1.0, m + 1, device="cuda", dtype=torch.float64)
    y, x = torch.meshgrid(ax, ax, indexing="ij")
    z = 1.0 - x.abs() - y.abs()
    fx = torch.where(z < 0, (1.0 - y.abs()) * torch.where(x < 0, -1.0, 1.0), x)
    fy = torch.where(z < 0, (1.0 - x.abs()) * torch.where(y < 0, -1.0, 1.0), y)
    p = _unit(torch.stack([fx, fy, z], -1).reshape(-1, 3))
    noise = _uniform(g, 1, 1, 9, 9, 9, lo=-1.0, hi=1.0)
    r = torch.nn.functional.grid_sample(noise, (p / 1.5).view(1, 1, 1, -1, 3),
                                        align_corners=True).reshape(-1)
    verts = (p * (1.0 + amplitude * r)[:, None]).to(torch.float32)
    c = torch.arange(m, device="cuda")
    a = (c[:, None] * (m + 1) + c[None, :]).reshape(-1)
    quad = torch.stack([a, a + 1, a + m + 2, a, a + m + 2, a + m + 1], 1)
    return verts, quad.reshape(-1, 3)[:faces].to(torch.int32).contiguous()


def _tet_grid(cells, g):
    """cells^3 jittered grid cells in the unit cube, five tetrahedra each, ordered so
    that the entering face comes first, and a scalar per vertex."""
    n1 = cells + 1
    ax = torch.arange(n1, device="cuda")
    q = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    p = q.double() / cells
    inner = ((q > 0) & (q < cells)).all(1, keepdim=True)
    p = p + inner * _uniform(g, *p.shape, lo=-0.2 / cells, hi=0.2 / cells)
    c = torch.arange(cells, device="cuda")
    c = torch.stack(torch.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    off = torch.tensor([[k & 1, (k >> 1) & 1, k >> 2] for k in range(8)], device="cuda")
    k = c[:, None] + off[None]
    corner = (k[..., 0] * n1 + k[..., 1]) * n1 + k[..., 2]
    even = torch.tensor([[0, 1, 2, 4], [3, 2, 1, 7], [5, 4, 7, 1], [6, 7, 4, 2], [1, 2, 4, 7]],
                        device="cuda")
    odd = torch.tensor([[1, 0, 5, 3], [2, 3, 6, 0], [4, 5, 0, 6], [7, 6, 3, 5], [0, 3, 5, 6]],
                       device="cuda")
    parity = (c.sum(1) & 1)[:, None, None]
    tets = torch.where(parity == 0, corner[:, even], corner[:, odd]).reshape(-1, 4)
    e = [p[tets[:, j]] - p[tets[:, 0]] for j in (1, 2, 3)]
    flip = (torch.linalg.cross(e[0], e[1]) * e[2]).sum(1) > 0
    tets = torch.where(flip[:, None], tets[:, [0, 2, 1, 3]], tets)
    cen, wid, amp = (_uniform(g, 4, 3, lo=0.2, hi=0.8), _uniform(g, 4, lo=0.1, hi=0.3),
                     _uniform(g, 4, lo=0.5, hi=1.0))
    s = sum(amp[j] * torch.exp(-((p - cen[j]) ** 2).sum(1) / (2 * wid[j] ** 2))
            for j in range(4))
    return p, tets.to(torch.int32).contiguous(), s.float()


def _rays(org, dirs):
    r = torch.zeros(dirs.shape[0], 8, device="cuda")
    r[:, 0:3] = org.float()
    r[:, 4:7] = dirs.float()
    r[:, 3] = torch.tensor([-1], dtype=torch.int32, device="cuda").view(torch.float32)
    return r


def _pinhole(width, height, eye, look, fov):
    """One ray per pixel centre, row by row, as a camera hands them over."""
    eye = torch.tensor(eye, device="cuda", dtype=torch.float64)
    look = _unit(torch.tensor(look, device="cuda", dtype=torch.float64) - eye)
    up = torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64)
    u = _unit(torch.linalg.cross(look, up))
    v = _unit(torch.linalg.cross(look, u))
    flen = 0.5 * height / math.tan(0.5 * math.radians(fov))
    px = torch.arange(width, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * width
    py = torch.arange(height, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * height
    d = flen * look + px[None, :, None] * u + py[:, None, None] * v
    return _rays(eye, _unit(d).reshape(-1, 3))


def _ortho(width, height, z):
    x = (torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width
    y = (torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height
    gy, gx = torch.meshgrid(y, x, indexing="ij")
    o = torch.stack([gx, gy, torch.full_like(gx, z)], -1).reshape(-1, 3)
    return _rays(o, torch.tensor([0.0, 0.0, -1.0], device="cuda").expand(o.shape[0], 3))


def _batch_sizes(case):
    """Faces and image side of each scene: the case's own, whatever the seed."""
    r = np.random.default_rng([7, case["scenes"], case["faces"]])
    hi = case["faces"]
    counts = np.exp(r.uniform(math.log(1e3), math.log(hi), case["scenes"])).astype(np.int64)
    counts[0] = hi
    counts = np.maximum(counts, 1024)
    sides = r.choice([s for s in (128, 256, 512, 1024) if s <= case["side"]], case["scenes"])
    sides[0] = case["side"]
    return counts, sides


def _blobs(res, g, shift=0.0):
    """A sum of 32 anisotropic Gaussian blobs scaled to peak below one."""
    cen = _uniform(g, 32, 3, lo=0.2, hi=0.8) + shift / (res - 1)
    sig, amp = _uniform(g, 32, 3, lo=0.03, hi=0.12), _uniform(g, 32, lo=0.3, hi=0.9)
    x = torch.linspace(0.0, 1.0, res, device="cuda", dtype=torch.float64)
    e = torch.exp(-0.5 * ((x[None, None] - cen[..., None]) / sig[..., None]) ** 2)
    out = torch.einsum("b,bz,by,bx->zyx", amp, e[:, 2], e[:, 1], e[:, 0])
    return (out * min(1.0, 0.95 / float(out.max()))).float().contiguous()


def _volume_inputs(case, seed):
    res = case["res"]
    density = _blobs(res, _generator(seed))
    tf = torch.as_tensor(S.transfer_function(256, seed=seed), device="cuda")
    target = None
    if case["backward"]:  # the image of another volume
        other = _blobs(res, _generator(seed), shift=2.0)
        target = V.march(other, tf, V.camera(case["width"], case["height"], res=res))[0]
    table = S.exp_coord_map(res + 1) if case["remap"] else None
    return density, tf, target, table


def _texture_inputs(case, seed):
    blocks, pool, gdim = S.sparse_pages(case["pages"], case["page"], seed=seed)
    g = _generator(seed)
    w, h, n = case["width"], case["height"], case["steps"]
    x = 0.8 * (torch.arange(w, device="cuda") + 0.5) / w
    y = 0.9 * (torch.arange(h, device="cuda") + 0.5) / h
    s = (torch.arange(n, device="cuda") + float(_uniform(g, 1))) / n
    uvw = torch.empty(h, w, n, 3, device="cuda")
    uvw[..., 0] = x[None, :, None] + 0.2 * s
    uvw[..., 1] = y[:, None, None] + 0.1 * s
    uvw[..., 2] = 1.0 - s
    return blocks, pool, gdim, uvw.reshape(-1, 3)


def _scene_accels(seed):
    g = _generator(seed)
    v, f = _sphere_mesh(131072, g)
    tri = TriangleAccel()
    tri.Build32(Mesh(v, f))
    n = 1000000
    pos = _uniform(g, n, 3).float()
    rad = (0.004 * torch.exp(0.5 * torch.randn(n, generator=g, device="cuda"))).float()
    sph = ParticleAccel()
    sph.Build32(Particles(pos, rad))
    p, t, _ = _tet_grid(32, g)
    tet = TetraAccel()
    tet.Build32(Tetrahedron(p.float(), t))
    return [(tri, (0.0, 0.0, 0.0), 2.2), (sph, (0.5, 0.5, 0.5), 1.0),
            (tet, (0.5, 0.5, 0.5), 1.0)]


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    """What a program holds before the call: inputs on the GPU and the handles it keeps."""
    kind, g = case["kind"], _generator(seed)
    if kind == "triangles":
        v, f = _sphere_mesh(case["faces"], g)
        return dict(case=case, accel=TriangleAccel(), mesh=Mesh(v, f),
                    rays=_pinhole(case["width"], case["height"], (0.1, 0.2, 3.0), (0, 0, 0), 45))
    if kind == "tetrahedra":
        p, t, s = _tet_grid(case["cells"], g)
        return dict(case=case, accel=TetraAccel(), scalar=s,
                    mesh=Tetrahedron(p if case["double"] else p.float(), t),
                    rays=_ortho(case["width"], case["height"], 2.0))
    if kind == "spheres":
        n = case["count"]
        median = 1e-3 * (16777216 / n) ** (1 / 3)
        pos = _uniform(g, n, 3).float()
        rad = (median * torch.exp(0.5 * torch.randn(n, generator=g, device="cuda"))).float()
        return dict(case=case, accel=ParticleAccel(), particles=Particles(pos, rad), seed=seed,
                    bounce=torch.zeros(case["width"] * case["height"], 4, device="cuda"),
                    rays=_pinhole(case["width"], case["height"], (0.5, 0.5, 2.2),
                                  (0.5, 0.5, 0.5), 30))
    if kind == "batch":
        counts, sides = _batch_sizes(case)
        verts, faces, rays, base = [], [], [], 0
        for n, side in zip(counts.tolist(), sides.tolist()):
            v, f = _sphere_mesh(n, g)
            verts.append(v)
            faces.append(f + base)
            rays.append(_pinhole(side, side, (0, 0, 3), (0, 0, 0), 45))
            base += v.shape[0]
        return dict(case=case, batch=TriangleBatch(), verts=torch.cat(verts),
                    faces=torch.cat(faces), rays=torch.cat(rays),
                    face_offsets=np.concatenate([[0], np.cumsum(counts)]),
                    ray_offsets=np.concatenate([[0], np.cumsum(sides.astype(np.int64) ** 2)]))
    if kind == "volume":
        density, tf, target, table = _volume_inputs(case, seed)
        if case["backward"]:
            density.requires_grad_(True)
            tf.requires_grad_(True)
        sampling = (V.Sampling(remap=(None, table, None), clamp=(False,) * 3)
                    if table is not None else None)
        return dict(case=case, density=density, tf=tf, target=target, sampling=sampling,
                    params=V.camera(case["width"], case["height"], res=case["res"]))
    if kind == "scene":
        accels, r, n = _scene_accels(seed), np.random.default_rng([31, seed]), case["grid"]
        graph = RenderGraph()
        for j in range(n ** 3):
            accel, centre, size = accels[j % 3]
            cell = np.array(np.unravel_index(j, (n,) * 3), np.float64) * 3.0 - 1.5 * (n - 1)
            to_origin = np.eye(4)
            to_origin[3, :3] = -np.asarray(centre)
            graph.AddRenderElement(accel, to_origin @ S.affine(
                r.normal(size=3), r.uniform(0, 360), (2.0 / size * r.uniform(0.8, 1.2),) * 3,
                cell + r.uniform(-0.3, 0.3, size=3)))
        s = (n + 1) / 5
        return dict(case=case, graph=graph, accels=accels,
                    camera=make_camera(case["side"], case["side"],
                                       eye=(-14.0 * s, 10.0 * s, 18.0 * s), fov=40.0))
    if kind == "lines":
        pos, seg, rad = S.line_strands(case["strands"], case["segments"], seed=seed)
        accel = LineAccel()
        accel.Build(Lines(torch.as_tensor(pos, device="cuda"),
                          torch.as_tensor(seg.astype(np.int32), device="cuda"),
                          torch.as_tensor(rad, device="cuda")))
        return dict(case=case, accel=accel,
                    rays=_pinhole(case["width"], case["height"], (0.3, 0.5, 3.4), (0, 0, 0), 40))
    if kind == "solids":
        v, ix = S.solid_grid(case["verts"], case["cells"], seed=seed)
        return dict(case=case, accel=SolidAccel(),
                    solids=Solid(case["verts"], torch.as_tensor(v, device="cuda"),
                                 torch.as_tensor(ix.astype(np.int32), device="cuda")),
                    rays=_pinhole(case["width"], case["height"], (1.7, 1.3, 2.1),
                                  (0.5, 0.5, 0.5), 50))
    blocks, pool, gdim, uvw = _texture_inputs(case, seed)
    tex = Texture3D()
    tex.set_sparse(blocks, pool, 0, 1, gdim)
    return dict(case=case, tex=tex, uvw=uvw)


def _hits(h):
    return {"t": h[:, 0], "uv": h[:, 1:3], "prim": h.view(torch.int32)[:, 3]}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "triangles":
        state["accel"].Build32(state["mesh"])
        if not case["isect"]:
            return _hits(state["accel"].Traverse(state["rays"]))
        r = state["accel"].Traverse(state["rays"], want_isect=True)
        x = r.isect.view(-1, 5, 4)
        return {**_hits(r.hits), "frame": x[:, :4, :3], "d": x[:, 4],
                "ids": x.view(torch.int32)[:, :4, 3]}
    if kind == "tetrahedra":
        state["accel"].Build32(state["mesh"])
        r = state["accel"].Traverse(state["rays"], want_subface=True, want_scalar=True,
                                    vertex_scalar=state["scalar"])
        return {**_hits(r.hits), "subface": r.subface, "scalar": r.scalar}
    if kind == "spheres":
        accel, rays = state["accel"], state["rays"]
        accel.Build32(state["particles"])
        r = accel.Traverse(rays, want_normal=True)
        more, normals = spawn_secondary(rays, r.hits, r.normal, state["seed"])
        bounce = state["bounce"]  # as many hits as primary rays hit something
        accel.Traverse(more, hits=bounce[:more.shape[0]], prev_normals=normals)
        return {"first": _hits(r.hits), "normal": r.normal, "second": _hits(bounce)}
    if kind == "batch":
        return _hits(state["batch"].build_trace(state["verts"], state["faces"],
                                                state["face_offsets"], state["rays"],
                                                state["ray_offsets"]))
    if kind == "volume":
        if not case["backward"]:
            return V.march(state["density"], state["tf"], state["params"],
                           sampling=state["sampling"])
        img = V.render(state["density"], state["tf"], state["params"], state["sampling"])
        loss = ((img - state["target"]) ** 2).sum()
        gd, gt = torch.autograd.grad(loss, (state["density"], state["tf"]))
        return {"image": img, "density_grad": gd, "tf_grad": gt}
    if kind == "scene":
        graph, cam = state["graph"], state["camera"]
        graph.Build()
        rays, pixel = camera_rays(cam)
        hits, element = graph.Trace(rays)
        colour, depth = framebuffer_write(cam, hits, pixel)
        return {**_hits(hits), "element": element, "colour": colour, "depth": depth}
    if kind == "lines":
        hits, normal = state["accel"].Traverse(state["rays"], want_normal=True)
        return {**_hits(hits), "normal": normal}
    if kind == "solids":
        state["accel"].Build32(state["solids"])
        hits, normal, position = state["accel"].Traverse(state["rays"], want_point=True)
        return {**_hits(hits), "normal": normal, "position": position}
    return state["tex"].Fetch(state["uvw"])


def _volume_samples(case):
    o, d, t0, t1 = _volume_rays(case)
    step = float(np.float32(0.5 * 2.0 / (case["res"] - 1)))
    return float(((t1 - t0) / step).floor().clamp(0, 8192).sum())


def work(case):
    """What a pass cannot do without: each input read once, each output written once,
    and for the traces one descent of the tree (two box tests a level) per ray."""
    kind = case["kind"]
    rays = case.get("width", 0) * case.get("height", 0)

    def descent(n, rays):
        return rays * 2 * 20 * math.log2(max(n, 2))

    if kind == "triangles":
        n = case["faces"]
        return {"bytes": 18 * n + rays * (32 + 16 + (80 if case["isect"] else 0)),
                "flops": descent(n, rays) + 30 * n}
    if kind == "tetrahedra":
        n, nv = 5 * case["cells"] ** 3, (case["cells"] + 1) ** 3
        return {"bytes": 16 * n + nv * (4 + (24 if case["double"] else 12)) + rays * (32 + 24),
                "flops": descent(n, rays) + 30 * n}
    if kind == "spheres":
        n = case["count"]
        return {"bytes": 16 * n + rays * (32 + 16 + 12 + 32 + 12 + 16),
                "flops": descent(n, 2 * rays) + 30 * n}
    if kind == "batch":
        counts, sides = _batch_sizes(case)
        nr = int((sides.astype(np.int64) ** 2).sum())
        return {"bytes": 18 * int(counts.sum()) + 48 * nr,
                "flops": sum(descent(int(n), int(s) ** 2) for n, s in zip(counts, sides))}
    if kind == "volume":
        samples = _volume_samples(case)
        vox = 4 * case["res"] ** 3
        if case["backward"]:
            return {"bytes": 3 * vox + rays * 60, "flops": 160 * samples}
        return {"bytes": vox + rays * 20, "flops": 60 * samples}
    if kind == "scene":
        rays = case["side"] ** 2
        return {"bytes": rays * (32 + 4 + 16 + 4 + 8), "flops": descent(1000000, rays)}
    if kind == "lines":
        n = case["strands"] * case["segments"]
        return {"bytes": 32 * n + rays * (32 + 16 + 12), "flops": descent(n, rays)}
    if kind == "solids":
        n = case["cells"] ** 3 * {8: 1, 6: 2, 5: 6}[case["verts"]]
        return {"bytes": 4 * case["verts"] * n + 12 * (case["cells"] + 1) ** 3
                + rays * (32 + 16 + 24), "flops": descent(n, rays) + 30 * n}
    n = rays * case["steps"]
    return {"bytes": n * (12 + 16 + 1), "flops": 12 * n}


# ---------------------------------------------------------------- in 64 bits
def _exact_triangles(case, seed):
    """Every ray against every triangle: the products of Moeller and Trumbore's test as
    dot products of the ray's and the triangle's Pluecker terms."""
    state = prepare(case, seed)
    v, f = state["mesh"].vertices.double(), state["mesh"].faces.long()
    o, d = state["rays"][:, 0:3].double(), state["rays"][:, 4:7].double()
    p0 = v[f[:, 0]]
    e1, e2 = v[f[:, 1]] - p0, v[f[:, 2]] - p0
    n = torch.linalg.cross(e1, e2)
    tri_u = torch.cat([e2, -torch.linalg.cross(e2, p0)], 1).T.contiguous()
    tri_v = torch.cat([-e1, -torch.linalg.cross(p0, e1)], 1).T.contiguous()
    tri_t = torch.cat([n, -(p0 * n).sum(1, keepdim=True)], 1).T.contiguous()
    nt = (-n).T.contiguous()
    ray6 = torch.cat([torch.linalg.cross(o, d), d], 1)
    ray4 = torch.cat([o, torch.ones_like(o[:, :1])], 1)
    rows = max(1, int(2.0e8 / f.shape[0]))
    t, uv, prim = [], [], []
    for k in range(0, o.shape[0], rows):
        inv = 1.0 / (d[k:k + rows] @ nt)
        u = (ray6[k:k + rows] @ tri_u) * inv
        w = (ray6[k:k + rows] @ tri_v) * inv
        at = (ray4[k:k + rows] @ tri_t) * inv
        at = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (at >= 0), at, math.inf)
        best, j = at.min(1)
        hit = torch.isfinite(best)
        t.append(torch.where(hit, best, FLT_MAX))
        uv.append(torch.where(hit[:, None], torch.stack([u.gather(1, j[:, None])[:, 0],
                                                         w.gather(1, j[:, None])[:, 0]], 1), 0.0))
        prim.append(torch.where(hit, j, -1))
    return {"t": torch.cat(t), "uv": torch.cat(uv), "prim": torch.cat(prim)}


def _volume_rays(case):
    """The shader camera's rays and where they cross the cube, in 64 bits."""
    w, h = case["width"], case["height"]
    flen = 0.5 * h / math.tan(0.5 * 45.0 * 3.14 / 180.0)
    x = torch.arange(w, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * w
    y = torch.arange(h, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * h
    gy, gx = torch.meshgrid(y, x, indexing="ij")
    # eye (0, 0, 3) looking down -z: u = +x, v = look x u = -y
    d = _unit(torch.stack([gx, -gy, torch.full_like(gx, -flen)], -1).reshape(-1, 3))
    o = torch.tensor([0.0, 0.0, 3.0], device="cuda", dtype=torch.float64)
    a, b = (-1.0 - o) / d, (1.0 - o) / d
    t0 = torch.minimum(a, b).max(1).values
    t1 = torch.maximum(a, b).min(1).values
    return o, d, t0, torch.maximum(t0, t1)


def _exact_march(case, density, tf, table, o, d, t0, t1):
    """Front-to-back emission and absorption along some rays: image rows and transmittance."""
    res, step = density.shape[0], float(np.float32(0.5 * 2.0 / (case["res"] - 1)))
    ns = ((t1 - t0) / step).floor().clamp(0, 8192)
    n = max(1, int(ns.max()))
    s = torch.arange(n, device="cuda", dtype=torch.float64)
    t = t0[:, None] + (s + 0.5) * step
    p = o + t[..., None] * d[:, None]
    live = (s < ns[:, None]) & ((p >= -1) & (p < 1)).all(-1)
    q = 0.5 * p + 0.5
    if table is not None:
        k = (q[..., 1].float() * table.numel()).long().clamp(0, table.numel() - 1)
        q = torch.stack([q[..., 0], table[k], q[..., 2]], -1)
        q = q - q.floor()
    q = q.clamp(0, 1) * (res - 1)
    c = q.floor().clamp(0, res - 1).long()
    f = q - c
    e = (c + 1).clamp(max=res - 1)
    rho = 0
    for z in (0, 1):
        for y in (0, 1):
            for x in (0, 1):
                at = [(e if b else c)[..., a] for a, b in ((0, x), (1, y), (2, z))]
                w = [(f if b else 1 - f)[..., a] for a, b in ((0, x), (1, y), (2, z))]
                rho = rho + (w[0] * w[1] * w[2] *
                             density.reshape(-1)[(at[2] * res + at[1]) * res + at[0]])
    top = tf.shape[0] - 1
    x = (rho * top).clamp(0, top)
    i = x.detach().floor().long().clamp(max=top)
    fr = (x - i)[..., None]
    rgba = (1 - fr) * tf[i] + fr * tf[(i + 1).clamp(max=top)]
    alpha = (1 - torch.exp(-20.0 * rgba[..., 3] * step)).clamp(max=float(np.float32(0.99)))
    alpha = torch.where(live, alpha, torch.zeros_like(alpha))
    T = torch.cumprod(1 - alpha, 1)
    before = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)
    colour = ((before * alpha)[..., None] * rgba[..., :3]).sum(1)
    return torch.cat([colour, 1 - T[:, -1:]], 1), T[:, -1]


def _exact_volume(case, seed):
    density, tf, target, table = _volume_inputs(case, seed)
    density, tf = density.double(), tf.double()
    table = None if table is None else torch.as_tensor(table, device="cuda").double()
    o, d, t0, t1 = _volume_rays(case)
    grad = case["backward"]
    if grad:
        density.requires_grad_(True)
        tf.requires_grad_(True)
        target = target.double().reshape(-1, 4)
    rows = max(1, int(6.0e6 / case["res"]) // 2)
    image, trans = [], []
    gd, gt = torch.zeros_like(density), torch.zeros_like(tf)
    for k in range(0, d.shape[0], rows):
        c = slice(k, k + rows)
        with torch.set_grad_enabled(grad):
            img, T = _exact_march(case, density, tf, table, o, d[c], t0[c], t1[c])
            if grad:
                a, b = torch.autograd.grad(((img - target[c]) ** 2).sum(), (density, tf))
                gd += a
                gt += b
        image.append(img.detach())
        trans.append(T.detach())
    image = torch.cat(image).view(case["height"], case["width"], 4)
    if grad:
        return {"image": image, "density_grad": gd, "tf_grad": gt}
    return image, torch.cat(trans).view(case["height"], case["width"])


def _exact_texture(case, seed):
    """The nearest texel of the page that holds the point; nothing between pages."""
    _, pool, gdim, uvw = _texture_inputs(case, seed)
    n, page = case["pages"], case["page"]
    pool = torch.from_numpy(np.frombuffer(pool, np.uint8).copy()).cuda()
    p = (uvw * torch.tensor(gdim, device="cuda", dtype=torch.float32)).double()
    f = p.floor().long()
    inside = ((p >= 0) & (p <= n * page)).all(1)
    f = f.clamp(0, n * page - 1)
    slot, at = f // page, f % page
    held = inside & ((slot.sum(1) & 1) == 0)
    z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda"),) * 3, indexing="ij")
    even = ((x + y + z) & 1) == 0
    rank = (torch.cumsum(even.reshape(-1), 0) - 1).view(n, n, n)
    k = rank[slot[:, 2], slot[:, 1], slot[:, 0]].clamp(min=0)
    texel = ((k * page + at[:, 2]) * page + at[:, 1]) * page + at[:, 0]
    v = torch.where(held, pool[texel].double() / 255.0, 0.0)
    out = torch.zeros(v.numel(), 4, device="cuda", dtype=torch.float64)
    out[:, 0] = v
    out[:, 3] = held
    return out


def exact(case, seed):
    """run()'s outputs in 64 bits.  The other accels' closest hits over millions of
    primitives have no value that every ray-primitive pair could be tried for in time."""
    if case["kind"] == "triangles" and not case["isect"]:
        if case["faces"] * case["width"] * case["height"] <= EXACT_PAIRS:
            return _exact_triangles(case, seed)
    if case["kind"] == "volume":
        return _exact_volume(case, seed)
    if case["kind"] == "texture":
        return _exact_texture(case, seed)
    return None
