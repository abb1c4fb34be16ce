"""The work this framework is used for, as cases that can be timed and compared.

Every case is a whole call of a user's program through the package's public entry points: the
draws, a plan's replay or a server's requests, and the read-back of what such a program reads
(the colour of a frame; all three planes where it picks or composites).  Sizes are those of the
tests and the benchmark: the reference application's 1000x600 window, the plain 512x512 frame, the
1920x1080 frame with a 2048^2 shadow map, the 4,000,000-triangle depth-order soup at 3840x2160,
and the serving mix (targets log-uniform over 128-3840 x 128-2160, six shaders, a shadow pass on
half of the requests).

A case's keys:
  kind      draw     one hsr.draw
            noalloc  one hsr.draw_noalloc
            frame    shadow pass + main pass in one hsr.draw_batch
            scene    several objects into one target, each after the ones before it, with a
                     shared shadow map, in one hsr.draw_batch
            plan     a recorded batch of `views` frames replayed with new uniforms
            serve    `views` requests through a render server
  mesh      sphere (displaced icosphere of subdivision `size`), split (the same with position, uv
            and normal indices of their own, as an OBJ file has), grid (height field of `size`^2
            cells), soup (`size` triangles), mixed (the serving pool)
  shader, width, height, shadow (side of a square shadow map, 0: none), bpp (bytes per texel of
  the diffuse map), tex (side of the textures), radius (the eye's distance), tile (the raster tile
  the program has chosen: 8 is the default, 16 what the autotuner takes for large batches),
  planes (color, or all three).
"""
import ctypes
import functools
import math
import os
import sys
import weakref

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "hana-softwarerenderer_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import hsr  # noqa: E402
from hsr import scenes, uniforms  # noqa: E402

SHADERS = ("ground", "toon", "texture", "texture_with_light", "blinn", "normalmap")
BLACK = (0, 0, 0, 255)


def listed():
    return [
        # a thumbnail of a small model: the smallest call, all three planes read (picking)
        _case("thumb_128", "draw", "grid", 32, "ground", 128, 128, planes="all"),
        # the plain frame: icosphere of 5,120 triangles, Blinn-Phong, no shadow
        _case("plain_512", "draw", "sphere", 4, "blinn", 512, 512, tex=256, radius=3.0),
        # the reference application's own window: an OBJ model with normal map and shadow
        _case("app_1000x600", "frame", "split", 4, "normalmap", 1000, 600, shadow=1000, bpp=3, tex=1024, radius=2.0),
        # a render loop that may not allocate, odd target size
        _case("noalloc_641x359", "noalloc", "sphere", 5, "texture", 641, 359, bpp=3, tex=509, radius=2.5, planes="all"),
        # the camera inside a model's bounds: faces crossing the frustum, large triangles
        _case("closeup_2560x1440", "draw", "sphere", 6, "texture_with_light", 2560, 1440, tex=1024, radius=1.12),
        # several objects in one target and one shadow map
        _case("scene_6_objects", "scene", "sphere", 4, "blinn", 1280, 720, shadow=1024, tex=512, radius=3.2, views=6),
        # the 1920x1080 frame: 327,680 triangles over a ground plane, 2048^2 shadow map
        _case("frame_1080p", "frame", "sphere", 7, "normalmap", 1920, 1080, shadow=2048, tex=1024, radius=3.2, plane=True),
        # an animation: one recorded frame replayed with a new camera
        _case("plan_720p", "plan", "grid", 256, "normalmap", 1280, 720, shadow=2048, tex=1024, radius=2.6, views=1),
        # a recorded batch of uneven views (contact sheet), replayed
        _case("plan_16_views", "plan", "mixed", 0, "mixed", 0, 0, views=16, tex=512, tile=16),
        # depth-order stress: overdraw of ~8, 1 in 100 triangles an exact duplicate
        _case("soup_4m_2160p", "draw", "soup", 4000000, "flat", 3840, 2160, tile=16, planes="all"),
        # one request to an idle server
        _case("serve_1", "serve", "mixed", 0, "mixed", 0, 0, views=1, tex=512, tile=16),
        # a busy server: a full batch of mixed requests over the resident pool
        _case("serve_64", "serve", "mixed", 0, "mixed", 0, 0, views=64, tex=1024, tile=16),
    ]


def _case(name, kind, mesh, size, shader, width, height, shadow=0, bpp=4, tex=256, radius=3.0, tile=8, views=1,
          planes="color", plane=False):
    return dict(name=name, kind=kind, mesh=mesh, size=size, shader=shader, width=width, height=height, shadow=shadow,
                bpp=bpp, tex=tex, radius=radius, tile=tile, views=views, planes=planes, plane=plane)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("draw", "draw", "noalloc", "frame", "frame", "scene", "plan", "plan", "serve", "serve"))
    c = _case("", kind, "mixed", 0, "mixed", 0, 0, tex=_log(rng, 64, 1024), bpp=rng.choice((1, 3, 4, 4)),
              radius=round(rng.uniform(1.1, 4.0), 3), tile=rng.choice((8, 8, 16, 16, 32)))
    del c["name"]
    if kind == "serve" or (kind == "plan" and rng.random() < 0.5):
        c["views"] = _log(rng, 1, 64 if kind == "serve" else 24)
        return c
    c["mesh"] = rng.choice(("sphere", "split", "grid") if kind != "draw" else ("sphere", "split", "grid", "soup"))
    if c["mesh"] == "soup":
        c["size"], c["shader"] = _log(rng, 10000, 3000000), "flat"
        c["width"], c["height"] = _log(rng, 256, 3840), _log(rng, 256, 2160)
        return c
    small = kind in ("noalloc", "scene")
    c["size"] = _log(rng, 16, 200 if small else 700) if c["mesh"] == "grid" else rng.randint(3, 5 if small else 7)
    c["shader"] = rng.choice(SHADERS)
    top = (1280, 720) if kind == "noalloc" else (3840, 2160)
    c["width"], c["height"] = _log(rng, 96, top[0]), _log(rng, 96, top[1])
    c["planes"] = rng.choice(("color", "color", "all"))
    if kind == "scene":
        c["views"] = rng.randint(2, 8)
    if kind in ("frame", "plan", "scene"):
        c["shadow"] = _log(rng, 200, 2048) if kind != "plan" or rng.random() < 0.6 else 0
        c["plane"] = kind == "frame" and rng.random() < 0.5
    return c


# ---- inputs ------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _icosphere(subdiv):
    """Unit icosphere (positions float64, triangles): the same for every seed, kept for the process."""
    return scenes.icosphere(subdiv)


def _normals(pos, tri):
    """Smooth unit normals (area-weighted face normals summed per vertex)."""
    a, b, c = (pos[tri[:, k]] for k in range(3))
    fn = np.cross(b - a, c - a)
    n = np.zeros_like(pos)
    for q in range(3):
        for k in range(3):
            n[:, q] += np.bincount(tri[:, k], weights=fn[:, q], minlength=len(pos))
    n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-30)
    return scenes.ref_normalize(n.astype(np.float32))


def _indexed(pos, nrm, uv, tri):
    faces = np.repeat(tri.astype(np.int32)[:, :, None], 3, axis=2)
    return scenes.Mesh(np.ascontiguousarray(pos, np.float32), nrm, np.ascontiguousarray(uv, np.float32), faces)


def _mesh(kind, size, seed, plane=False):
    rng = np.random.default_rng(seed)
    if kind == "soup":
        return _soup(size, rng)
    if kind == "grid":
        xs = np.linspace(-1, 1, size + 1)
        x, z = (v.ravel() for v in np.meshgrid(xs, xs))
        p = np.stack([x, np.zeros_like(x), z], 1)
        p[:, 1] = 0.15 * scenes.fbm(p, seed, octaves=3)
        i = np.arange((size + 1) ** 2).reshape(size + 1, size + 1)
        a, b, c, d = i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, 1:].ravel(), i[1:, :-1].ravel()
        tri = np.concatenate([np.stack([a, d, c], 1), np.stack([a, c, b], 1)])
        return _indexed(p, _normals(p, tri), np.stack([(x + 1) / 2, (z + 1) / 2], 1), tri)
    p, tri = _icosphere(size)
    pd = p * (1.0 + 0.05 * scenes.fbm(p, seed, octaves=3))[:, None]
    m = _indexed(pd, _normals(pd, tri), scenes.spherical_uv(p), tri)
    if kind == "split":  # uvs and normals in arrays of their own order
        for k, name in ((1, "uv"), (2, "nrm")):
            at = rng.permutation(len(p)).astype(np.int32)
            v = np.empty_like(getattr(m, name))
            v[at] = getattr(m, name)
            setattr(m, name, v)
            m.faces[:, :, k] = at[tri]
    return scenes.concat_meshes(m, scenes.ground_plane(-1.2, 6.0)) if plane else m


def _soup(n, rng):
    """Depth-order stress in NDC (identity transforms): counter-clockwise triangles of constant
    depth, lognormal edges with a median of 2 pixels of a 3840x2160 target, 1 in 100 an exact
    duplicate submitted later."""
    nb = n - n // 100
    cx, cy, z = (rng.random(nb, dtype=np.float32) for _ in range(3))
    edge = 2.0 * np.exp(1.06 * rng.standard_normal(nb, dtype=np.float32)) * math.sqrt(4000000 / n)
    r = (edge / math.sqrt(3.0)).astype(np.float32)
    th = rng.random(nb, dtype=np.float32) * np.float32(2 * math.pi)
    pos = np.empty((nb, 3, 3), np.float32)
    for k in range(3):
        t = th + np.float32(2 * math.pi * k / 3) + (rng.random(nb, dtype=np.float32) - np.float32(0.5)) * np.float32(0.7)
        pos[:, k, 0] = cx * 2 - 1 + r * np.cos(t) * np.float32(2 / 3840)
        pos[:, k, 1] = cy * 2 - 1 + r * np.sin(t) * np.float32(2 / 2160)
        pos[:, k, 2] = z
    tri = np.concatenate([np.arange(nb, dtype=np.int32), rng.integers(0, nb, n - nb, dtype=np.int32)])
    faces = np.zeros((n, 3, 3), np.int32)
    for k in range(3):
        faces[:, k, 0] = tri * 3 + k
    return scenes.Mesh(pos.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), np.zeros((1, 2), np.float32), faces)


# the serving pool: 3,302,400 triangles (benchmark's mesh kinds and sizes)
_POOL = (("sphere", 7), ("sphere", 7), ("grid", 512), ("grid", 800), ("grid", 512), ("sphere", 6), ("sphere", 6), ("grid", 256))
_POOL_SMALL = (("sphere", 6), ("grid", 128), ("sphere", 5), ("sphere", 7), ("grid", 256), ("grid", 32))


def _pool(case):
    return _POOL if case["views"] > 16 else _POOL_SMALL


def _views(case):
    """The frames of a plan or a server's batch: (mesh number, shader, width, height, shadow side).
    A mixed batch draws them from the serving mix, the same for every seed: a recorded
    batch keeps its targets, and a stream keeps its mix."""
    if case["mesh"] != "mixed":
        return [(0, case["shader"], case["width"], case["height"], case["shadow"])] * case["views"]
    rng = np.random.default_rng(1000 + case["views"] * 31 + case["tex"])
    top = (3840, 2160) if case["kind"] == "serve" else (1920, 1080)
    out = []
    for _ in range(case["views"]):
        m = int(rng.integers(len(_pool(case))))
        w = int(round(math.exp(rng.uniform(math.log(128), math.log(top[0])))))
        h = int(round(math.exp(rng.uniform(math.log(128), math.log(top[1])))))
        out.append((m, SHADERS[int(rng.integers(6))], w, h, scenes.serve_shadow_size(w, h) if rng.random() < 0.5 else 0))
    return out


def _eye(rng, kind, radius, orbit=False):
    """A camera around the origin: anywhere (`orbit`), or on the side that the light at (2, 2, 2) is on."""
    el = rng.uniform(0.35, 1.1) if kind == "grid" else rng.uniform(-0.3, 0.7)
    az = rng.uniform(0, 2 * math.pi) if orbit else rng.uniform(0.1, 1.4)
    return (radius * math.cos(el) * math.sin(az), radius * math.sin(el), radius * math.cos(el) * math.cos(az))


def _pinned(shape, dtype):
    """Page-locked array (hsr_host_alloc); the memory is given back when the last view of it goes."""
    held = hsr.PinnedArray((int(np.prod(shape)),), dtype)
    a, held.array = held.array, None
    root = a
    while isinstance(root.base, np.ndarray):
        root = root.base
    weakref.finalize(root, hsr.lib().hsr_host_free, ctypes.c_void_p(held.ptr))
    return a.reshape(shape)


class State:
    """What the program holds between calls; released when the last reference goes."""

    def __init__(self):
        self.held, self.server, self.plan = [], None, None

    def hold(self, x):
        self.held.append(x)
        return x

    def __del__(self):
        if self.server is not None:
            self.server.close()
        if self.plan is not None:
            self.plan.release()
        for x in reversed(self.held):
            x.release()


def prepare(case, seed):
    hsr.init(0)
    hsr.set_tuning(tile=case["tile"], warps_per_cta=4, ctas_per_sm=8, bin_factor=4.0)
    rng = np.random.default_rng(seed)
    s = State()
    s.kind = case["kind"]
    t = case["tex"]
    nmap = scenes.normal_map_texture(t, t, seed + 2)
    dif, nrm = s.hold(hsr.Texture(scenes.noise_texture(t, t, case["bpp"], seed + 1))), s.hold(hsr.Texture(nmap))
    if case["kind"] in ("plan", "serve"):
        spec = _pool(case) if case["mesh"] == "mixed" else ((case["mesh"], case["size"]),)
        views = _views(case)
        used = {m for m, *_ in views}
        meshes = {m: s.hold(hsr.Mesh(_mesh(k, z, seed * 64 + m))) for m, (k, z) in enumerate(spec) if m in used}
        eyes = [_eye(rng, spec[m][0], rng.uniform(2.0, 4.0) if case["mesh"] == "mixed" else case["radius"], case["mesh"] == "mixed") for m, *_ in views]
        sds = [hsr.shader_data_build(e, w, h, enable_shadow=sh > 0) for e, (m, _, w, h, sh) in zip(eyes, views)]
        s.out = _pinned((sum(w * h * 4 for _, _, w, h, _ in views),), np.uint8)
        s.outs, at = [], 0
        for _, _, w, h, _ in views:
            s.outs.append(s.out[at:at + w * h * 4].reshape(h, w, 4))
            at += w * h * 4
        if case["kind"] == "serve":
            s.server = hsr.Server(pool_bytes=40 << 30, max_batch=64, slots=2)
            s.asks = [dict(mesh=meshes[m], shader=scenes.SHADER_NAMES.index(n), sd=sd, width=w, height=h, diffuse=dif,
                           normal=nrm, shadow_size=sh, out={"color": o}) for (m, n, w, h, sh), sd, o in zip(views, sds, s.outs)]
            return s
        s.sets, s.targets, descs = [], [], []
        for (m, n, w, h, sh), sd in zip(views, sds):
            main = s.hold(hsr.Target(w, h))
            smap = s.hold(hsr.Target(sh, sh)) if sh else None
            if smap:
                s.sets.append((len(descs), sd))
                descs.append(hsr.make_desc(meshes[m], scenes.SHADOW, sd, smap, dif, nrm, clear=(BLACK, scenes.FLT_MAX)))
            s.sets.append((len(descs), sd))
            descs.append(hsr.make_desc(meshes[m], scenes.SHADER_NAMES.index(n), sd, main, dif, nrm, shadow_map=smap,
                                       clear=(BLACK, scenes.FLT_MAX)))
            s.targets.append(main)
        s.plan = hsr.Plan(descs)
        return s
    w, h, shadow = case["width"], case["height"], case["shadow"]
    shader = scenes.SHADER_NAMES.index(case["shader"])
    main = s.target = s.hold(hsr.Target(w, h))
    smap = s.hold(hsr.Target(shadow, shadow)) if shadow else None
    names = (("color", np.uint8, (h, w, 4)), ("depth", np.float32, (h, w)), ("prim", np.uint32, (h, w)))
    s.planes = {k: _pinned(shape, dt) for k, dt, shape in names if case["planes"] == "all" or k == "color"}
    # primitive ids as int32: numpy's uint32 has few operations in torch
    s.result = {k: v.view(np.int32) if k == "prim" else v for k, v in s.planes.items()}
    s.keep = []  # uniforms stay alive with the descriptors
    clear = (BLACK, 1.0)

    def desc(mesh, sh, sd, target, sm=None, base=0, first=True):
        return hsr.make_desc(mesh, sh, sd, target, dif, nrm, shadow_map=sm, prim_base=base, clear=clear if first else None, keep=s.keep)

    objects = case["views"] if case["kind"] == "scene" else 1
    eye = _eye(rng, case["mesh"], case["radius"])
    descs, mains, base = [], [], 0
    for k in range(objects):
        mesh = s.hold(hsr.Mesh(_mesh(case["mesh"], case["size"], seed * 16 + k, case["plane"])))
        if case["mesh"] == "soup":
            sd = uniforms.shader_data((0, 0, 1), w, h, identity_mvp=True)
        else:
            place = hsr.transform(position=rng.uniform(-0.9, 0.9, 3), scale=[float(rng.uniform(0.3, 0.8))] * 3) if objects > 1 else None
            sd = hsr.shader_data_build(eye, w, h, model=place, enable_shadow=shadow > 0)
        if smap:
            descs.append(desc(mesh, scenes.SHADOW, sd, smap, first=k == 0))
        mains.append(desc(mesh, shader, sd, main, smap, base, k == 0))
        base += mesh.nfaces
    s.descs = descs + mains
    return s


def run(state):
    s = state
    if s.kind == "serve":
        tickets = [s.server.submit(**a) for a in s.asks]
        for t in tickets:
            if s.server.wait(t)["status"] != hsr.OK:
                raise RuntimeError("a request failed")
        return s.out
    if s.kind == "plan":
        for k, sd in s.sets:
            s.plan.set_uniforms(k, sd)
        s.plan.launch()
        s.plan.wait()
        for t, o in zip(s.targets, s.outs):
            t.download(depth=False, prim=False, out={"color": o})
        return s.out
    if s.kind == "draw":
        hsr.draw(s.descs[0])
    elif s.kind == "noalloc":
        hsr.draw_noalloc(s.descs[0])
    else:
        hsr.draw_batch(s.descs)
    s.target.download(depth="depth" in s.planes, prim="prim" in s.planes, out=s.planes)
    return s.result


def exact(case, seed):
    """None: a frame's colours and primitive ids are whole numbers, and its depths have no value in
    64 bits of their own.  Which triangle a pixel's depth comes from is decided by single-precision
    edge tests, part of the contract (bit for bit the reference's), which 64 bits decide
    otherwise along every edge."""
    return None


# ---- what a pass cannot do without ---------------------------------------------------------
def _mesh_counts(kind, size):
    """(positions, faces, bytes): positions, normals and uvs once, and the face indices."""
    if kind == "soup":
        return (size - size // 100) * 3, size, (size - size // 100) * 36 + size * 12
    v, f = ((size + 1) ** 2, 2 * size * size) if kind == "grid" else (10 * 4 ** size + 2, 20 * 4 ** size)
    return v, f, v * 32 + f * (36 if kind == "split" else 12)


def work(case):
    """Bytes: each mesh once per pass over it, the texels once (no more than one per pixel), each
    target plane that the caller can read written once and each plane read back read once.
    Operations: 28 per position (the 4x4 product), 60 per face (cull and setup), 150 per
    pixel (coverage, depth, shading)."""
    nbytes = flops = 0
    mixed = case["mesh"] == "mixed"
    multi = case["kind"] in ("plan", "serve")
    views = _views(case) if multi else [(0, case["shader"], case["width"], case["height"], case["shadow"])]
    spec = _pool(case) if mixed else ((case["mesh"], case["size"]),)
    objects = case["views"] if case["kind"] == "scene" else 1
    for m, shader, w, h, sh in views:
        v, f, b = _mesh_counts(*spec[m])
        passes = (2 if sh else 1) * objects
        px, spx = w * h, sh * sh
        texels = min(px, case["tex"] ** 2) * ((case["bpp"] + 3 * (shader == "normalmap")) if shader not in ("ground", "toon", "flat") else 0)
        # a served request's depth and primitive ids are not asked for, nor is its shadow map's
        plane = 4 if case["kind"] == "serve" else 12
        back = 12 if case["planes"] == "all" else 4
        nbytes += passes * b + texels + px * (plane + back) + spx * (plane + 4)
        flops += passes * (28 * v + 60 * f) + 150 * px + 60 * spx
    return {"bytes": nbytes, "flops": flops}
