"""Timed workloads of the displaced-surface query, through its public entry points.

A case is a dict of plain values:

  kind     query    a device batch of rays (Scene.intersect_device)
           host     the same from host arrays (Scene.intersect)
           rebuild  a new height map: pyramid build, scene setup, one camera query
           render   the batched path tracer (Scene.render)
           serve    a burst of requests through the continuous-batching server
           mesh     the uniform oracle mesh into device buffers (dmap_tessellate_uniform)
  scene    quad     one unit quad (2 triangles) with one n x n map
           sphere   the cube sphere, 6 k^2 patches of two triangles, each patch its own map
                    (beyond 96 patches the patches share 32 maps, as a tiled texture does)
           ground   the sphere with a displaced ground plane of 2n x 2n texels and an emitter
  n, k     texels per map side, patches per cube face side
  texel    f32 or f16 height texels
  rays     ray count (kinds query, host, rebuild, serve), as drawn by `mix`
  mix      camera   jittered pinhole camera rays
           frame    camera rays and one cosine-weighted bounce per visible point (3 : 1)
           grazing  frame rays and rays 0.1-5 degrees above the base surface (3 : 1)
           shadow   from surface points toward the emitter, ending just before it

Height maps follow the benchmark's generator (seeded sines of 1-32 cycles a
tile plus octaves of value noise; a ridged multifractal for the ground); all
inputs are made on the GPU from the seed alone, none from a query's answers.
"""
import ctypes
import math

import numpy as np
import torch

import dmap_b200 as dm
from dmap_b200 import scenes

DEV = "cuda"
F8 = torch.float64
SHARED_MAPS = 32

_ctx = None


def context():
    """The process's device context; its calls all go to its own stream."""
    global _ctx
    if _ctx is None:
        _ctx = dm.Context(0)
    return _ctx


# ---- the cases -------------------------------------------------------------

def _case(name, kind, scene, n, rays, **more):
    c = {"name": name, "kind": kind, "scene": scene, "n": n, "k": 1 if scene == "quad" else 4, "texel": "f32",
         "rays": rays, "mix": "camera" if scene == "quad" else "frame", "mode": "closest", "order": "nearest",
         "leaf": "f32", "record": "f32", "graph": False}
    c.update(more)
    return c


def listed():
    return [
        # a pick or a probe from an application: a few rays, answered at once
        _case("pick", "host", "quad", 512, 64, record="f64"),
        # a small host batch per frame of an interactive tool, by graph replay
        _case("probe_graph", "host", "quad", 512, 4096, graph=True),
        # the small plain-method benchmark: 256 x 256 camera rays on one quad
        _case("quad_camera", "query", "quad", 512, 65536),
        # one tile of a bucket renderer: a ragged batch over the whole sphere
        _case("sphere_tile", "query", "sphere", 512, 20011),
        # the benchmark frame: 1920 x 1080 primaries and their bounces, 17 GB of pyramids
        _case("sphere_frame", "query", "sphere", 2048, 2796668),
        # the precision variant: FP16 texels and grazing rays
        _case("sphere_f16_grazing", "query", "sphere", 1024, 1500007, texel="f16", mix="grazing"),
        # next-event estimation: shadow rays of the path tracer's scene
        _case("shadow_rays", "query", "ground", 512, 1000003, mix="shadow", mode="occluded"),
        # the C++ adapter's defaults: double records, index order, the reference's FP64 leaf
        _case("adapter_f64", "host", "sphere", 512, 100003, record="f64", order="index", leaf="f64"),
        # a finely tessellated object: 12,288 triangles behind the triangle tree
        _case("many_triangles", "query", "sphere", 64, 700001, k=32),
        # a height map edited between frames: rebuild its pyramid, trace a preview
        _case("rebuild", "rebuild", "quad", 1024, 65536),
        # the path tracer at preview quality: 640 x 360, 4 samples per pixel, depth 5
        _case("render_preview", "render", "ground", 512, 640 * 360 * 4, width=640, height=360, spp=4),
        # a burst of requests of very different sizes, nine in ten of them closest-hit
        _case("serve_burst", "serve", "sphere", 512, 1200000, requests=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "query", "host", "host", "rebuild", "render", "serve", "mesh"])
    order = rng.choice(["nearest", "nearest", "nearest", "index"])
    leaf = rng.choice(["f32", "f32", "f32", "f64"])
    texel = rng.choice(["f32", "f32", "f16"])
    name = ""
    if kind == "rebuild":
        c = _case(name, kind, "quad", 2 ** rng.randint(6, 11), _log_int(rng, 64, 200000), texel=texel)
    elif kind == "render":
        w = 2 * _log_int(rng, 40, 480)
        h, spp = max(2, w * 9 // 16), rng.randint(1, 4)
        c = _case(name, kind, "ground", 2 ** rng.randint(7, 9), w * h * spp, width=w, height=h, spp=spp)
    elif kind == "serve":
        c = _case(name, kind, "sphere", 2 ** rng.randint(7, 9), _log_int(rng, 20000, 1500000),
                  requests=rng.randint(2, 40))
    elif kind == "mesh":
        c = _case(name, kind, rng.choice(["quad", "sphere"]), 2 ** rng.randint(7, 10), 0, sub=_log_int(rng, 3, 300))
    else:
        which = rng.choice(["quad", "sphere", "sphere", "fine", "ground"])
        rays = _log_int(rng, 1, 1000000) if kind == "query" else _log_int(rng, 1, 200000)
        if which == "quad":
            c = _case(name, kind, "quad", 2 ** rng.randint(6, 11), rays, mix=rng.choice(["camera", "frame"]))
        elif which == "fine":
            c = _case(name, kind, "sphere", 2 ** rng.randint(4, 6), rays, k=rng.randint(7, 40))
        elif which == "ground":
            c = _case(name, kind, "ground", 2 ** rng.randint(7, 9), rays, mix="shadow", mode="occluded")
        else:
            c = _case(name, kind, "sphere", 2 ** rng.randint(7, 10), rays, texel=texel,
                      mix=rng.choice(["camera", "frame", "grazing"]))
        c.update(order=order, leaf=leaf, record=rng.choice(["f32", "f32", "f64"]))
        c["graph"] = kind == "host" and rng.random() < 0.5
    del c["name"]
    return c


# ---- height maps -------------------------------------------------------------

def _weights(n, cells):
    """(n, cells + 1) smoothstep interpolation weights at s / (n - 1), s = 0..n-1."""
    x = torch.linspace(0.0, 1.0, n, dtype=F8, device=DEV) * cells
    i = x.floor().long().clamp_(max=cells - 1)
    f = x - i
    f = f * f * (3.0 - 2.0 * f)
    w = torch.zeros(n, cells + 1, dtype=F8, device=DEV)
    rows = torch.arange(n, device=DEV)
    w[rows, i] += 1.0 - f
    w[rows, i + 1] += f
    return w


def _noise(n, cells, rng):
    cells = min(cells, max(n - 1, 1))
    lat = torch.from_numpy(rng.uniform(-1.0, 1.0, (cells + 1, cells + 1))).to(DEV)
    w = _weights(n, cells)
    return w @ lat @ w.T


def _close(h):
    return torch.cat([torch.cat([h, h[:, -1:]], 1), torch.cat([h[-1:], h[-1:, -1:]], 1)], 0)


def _sines(n, rng, amplitude, octaves):
    """The benchmark's map: 8 plane waves (log-uniform 1-32 cycles, amplitude
    1/f) and value noise, scaled to max |h| = amplitude; (n + 1)^2 nodes."""
    u = (torch.arange(n, dtype=F8, device=DEV) + 0.5) / n
    f = torch.from_numpy(np.exp(rng.uniform(0.0, math.log(32.0), 8))).to(DEV)
    th, ph = (torch.from_numpy(rng.uniform(0.0, 2.0 * math.pi, 8)).to(DEV)[:, None] for _ in range(2))
    a = 2.0 * math.pi * f[:, None] * torch.cos(th) * u
    b = 2.0 * math.pi * f[:, None] * torch.sin(th) * u + ph
    inv = 1.0 / f[:, None]
    h = (torch.cos(b) * inv).T @ torch.sin(a) + (torch.sin(b) * inv).T @ torch.cos(a)
    h = h / h.abs().max()
    z = sum(_noise(n, 8 << o, rng) * 0.5 ** o for o in range(octaves))
    h = h + 0.35 * z / z.abs().max()
    return _close(h * (amplitude / h.abs().max()))


def _ridged(n, rng, amplitude):
    h = sum((1.0 - _noise(n, 4 << o, rng).abs()) ** 2 * 0.5 ** o for o in range(6))
    h = h - h.min()
    return _close(h * (amplitude / h.max()))


def _maps(case, seed):
    """The scene's node grids on the GPU, in the texel type."""
    dt = torch.float16 if case["texel"] == "f16" else torch.float32
    rng = np.random.Generator(np.random.PCG64(seed))
    n, k = case["n"], case["k"]
    if case["scene"] == "quad":
        return [_sines(n, rng, 0.05, 2).to(dt)]
    count = 6 * k * k if k <= 4 else SHARED_MAPS
    maps = [_sines(n, rng, 0.08 * 4.0 / max(k, 4), 4).to(dt) for _ in range(count)]
    if case["scene"] == "ground":
        maps.append(_ridged(2 * n, rng, 0.2).to(dt))
    return maps


# The cube's faces: outward normal and the (u, v) axes of its patches.
FACES = np.array([[[1, 0, 0], [0, 1, 0], [0, 0, 1]], [[-1, 0, 0], [0, 0, 1], [0, 1, 0]],
                  [[0, 1, 0], [0, 0, 1], [1, 0, 0]], [[0, -1, 0], [1, 0, 0], [0, 0, 1]],
                  [[0, 0, 1], [1, 0, 0], [0, 1, 0]], [[0, 0, -1], [0, 1, 0], [1, 0, 0]]], np.float64)


def _split(P, N):
    """Quads' corners and normals (m, 4, 3) in the order 00, 10, 01, 11 as two triangles each, (2 m, 24)."""
    out = np.zeros((len(P), 2, 24))
    for q, (corners, t) in enumerate((((0, 1, 2), (0, 0, 1, 0, 0, 1)), ((3, 2, 1), (1, 1, 0, 1, 1, 0)))):
        out[:, q, 0:9] = P[:, corners].reshape(-1, 9)
        out[:, q, 9:18] = N[:, corners].reshape(-1, 9)
        out[:, q, 18:24] = t
    return out.reshape(-1, 24)


def _flat(p00, p10, p01, p11, up):
    return _split(np.array([[p00, p10, p01, p11]], np.float64), np.tile(np.array(up, np.float64), (1, 4, 1)))


def _geometry(case):
    """Base triangles (t, 24) and each one's map."""
    if case["scene"] == "quad":
        return _flat((0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1)), np.zeros(2, np.int32)
    k = case["k"]
    b, a = (x.reshape(-1) for x in np.mgrid[0:k, 0:k])
    uv = np.stack([np.stack([a + p, b + q], 1) for q in (0, 1) for p in (0, 1)], 1) * (2.0 / k) - 1.0
    c = FACES[:, None, None, 0] + uv[None, ..., 0:1] * FACES[:, None, None, 1] + uv[None, ..., 1:2] * FACES[:, None,
                                                                                                         None, 2]
    c = (c / np.linalg.norm(c, axis=-1, keepdims=True)).reshape(-1, 4, 3)
    tris = _split(c, c)
    which = (np.arange(len(tris)) // 2).astype(np.int32)
    if k > 4:
        which = which % SHARED_MAPS
    if case["scene"] == "ground":
        y = -1.3
        tris = np.concatenate([tris, _flat((-2, y, 2), (2, y, 2), (-2, y, -2), (2, y, -2), (0, 1, 0))])
        which = np.concatenate([which, np.full(2, which.max() + 1, np.int32)])
    return tris, which


# ---- the surface in 64 bits: what the inputs and exact() need of it ---------

def _height(maps, which, st):
    """Bilinear heights and their gradients at st (m, 2) of maps[which]."""
    h = torch.zeros(len(st), dtype=F8, device=DEV)
    g = torch.zeros(len(st), 2, dtype=F8, device=DEV)
    for size in sorted({len(x) for x in maps}):
        ids = [q for q, x in enumerate(maps) if len(x) == size]
        flat = maps[ids[0]].reshape(-1) if len(ids) == 1 else None
        if flat is None:
            key = tuple(ids)
            flat = _stack(maps, key)
        slot = torch.full((len(maps),), -1, dtype=torch.long, device=DEV)
        slot[torch.tensor(ids, device=DEV)] = torch.arange(len(ids), device=DEV)
        here = slot[which]
        n = size - 1
        f = st.clamp(0.0, 1.0) * n
        c = f.long().clamp_(max=n - 1)
        s, t = (f - c).unbind(1)
        at = here.clamp(min=0) * (size * size) + c[:, 1] * size + c[:, 0]
        v00, v10, v01, v11 = (flat[at + d].double() for d in (0, 1, size, size + 1))
        ok = here >= 0
        h = torch.where(ok, (1 - s) * (1 - t) * v00 + s * (1 - t) * v10 + (1 - s) * t * v01 + s * t * v11, h)
        gr = torch.stack([((1 - t) * (v10 - v00) + t * (v11 - v01)) * n, ((1 - s) * (v01 - v00) + s * (v11 - v10)) * n],
                         1)
        g = torch.where(ok[:, None], gr, g)
    return h, g


_stacked = (None, None)


def _stack(maps, key):
    global _stacked
    if _stacked[0] is not maps or _stacked[1][0] != key:
        _stacked = (maps, (key, torch.stack([maps[q] for q in key]).reshape(-1)))
    return _stacked[1][1]


def _forget():
    global _stacked
    _stacked = (None, None)


def _charts(tris):
    """Per triangle, with texture coordinates (s, t): P = q0 + s e1 + t e2, M = m0 + s Mu + t Mv and
    barycentrics J ((s, t) - t0)."""
    T = torch.from_numpy(np.ascontiguousarray(tris)).to(DEV)
    p, m, t = T[:, 0:9].view(-1, 3, 3), T[:, 9:18].view(-1, 3, 3), T[:, 18:24].view(-1, 3, 2)
    J = torch.linalg.inv(torch.stack([t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]], 2))
    E = torch.stack([p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]], 2) @ J
    D = torch.stack([m[:, 1] - m[:, 0], m[:, 2] - m[:, 0]], 2) @ J
    q0 = p[:, 0] - (E @ t[:, 0, :, None])[..., 0]
    m0 = m[:, 0] - (D @ t[:, 0, :, None])[..., 0]
    return {"q0": q0, "e1": E[..., 0], "e2": E[..., 1], "m0": m0, "Mu": D[..., 0], "Mv": D[..., 1], "J": J,
            "t0": t[:, 0]}


def _surface(maps, which, charts, tri, st):
    """Point and unit normal of the displaced surface of triangles tri at st."""
    g = {k: v[tri] for k, v in charts.items()}
    s, t = st[:, 0:1], st[:, 1:2]
    P, M = g["q0"] + s * g["e1"] + t * g["e2"], g["m0"] + s * g["Mu"] + t * g["Mv"]
    ml = M.norm(dim=1, keepdim=True)
    N = M / ml
    Nu = (g["Mu"] - (N * g["Mu"]).sum(1, keepdim=True) * N) / ml
    Nv = (g["Mv"] - (N * g["Mv"]).sum(1, keepdim=True) * N) / ml
    h, gr = _height(maps, which[tri], st)
    h = h[:, None]
    ng = torch.linalg.cross(g["e1"] + gr[:, 0:1] * N + h * Nu, g["e2"] + gr[:, 1:2] * N + h * Nv)
    return P + h * N, ng / ng.norm(dim=1, keepdim=True)


# ---- rays ------------------------------------------------------------------

def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _frame_of(n):
    a = torch.zeros_like(n)
    small = n[:, 0].abs() < 0.9
    a[:, 0], a[:, 1] = small.double(), (~small).double()
    t1 = _unit(torch.linalg.cross(a, n))
    return t1, torch.linalg.cross(n, t1)


def _camera(case, m, gen):
    """m jittered pinhole rays in image rows, the image sized for them."""
    quad = case["scene"] == "quad"
    eye, at, aspect = ((0.5, 0.5, 2.0), (0.5, 0.5, 0.0), 1.0) if quad else ((0.9, 1.1, 2.6), (0.0, 0.0, 0.0), 16 / 9)
    eye, at, up = (torch.tensor(x, dtype=F8, device=DEV) for x in (eye, at, (0.0, 1.0, 0.0)))
    w = max(1, math.ceil(math.sqrt(m * aspect)))
    h = -(-m // w)
    f = (at - eye) / (at - eye).norm()
    r = torch.linalg.cross(f, up)
    r = r / r.norm()
    u = torch.linalg.cross(r, f)
    q = torch.arange(m, device=DEV)
    jit = torch.rand(m, 2, dtype=F8, device=DEV, generator=gen)
    th = math.tan(math.radians(22.5))
    px = ((q % w + jit[:, 0]) / w * 2.0 - 1.0) * th * aspect
    py = (1.0 - (q // w + jit[:, 1]) / h * 2.0) * th
    d = _unit(f + px[:, None] * r + py[:, None] * u)
    return eye.expand(m, 3), d, torch.full((m,), math.inf, dtype=F8, device=DEV)


def _points(m, n_tri, gen, last_share=0.0):
    """m random (triangle, st); last_share of them on the last two triangles."""
    tri = torch.randint(0, n_tri, (m,), device=DEV, generator=gen)
    if last_share > 0.0:
        on = torch.rand(m, device=DEV, generator=gen) < last_share
        tri = torch.where(on, n_tri - 1 - tri % 2, tri)
    st = torch.rand(m, 2, dtype=F8, device=DEV, generator=gen)
    fold = (st.sum(1) > 1.0) != (tri % 2 == 1)  # triangle 2p is s + t < 1, 2p + 1 the rest
    return tri, torch.where(fold[:, None], 1.0 - st, st)


def _rays(case, maps, tris, which, seed, m=None, mix=None):
    m, mix = m or case["rays"], mix or case["mix"]
    gen = torch.Generator(DEV).manual_seed(seed * 7919 + 17)
    charts, wh = _charts(tris), torch.from_numpy(which).to(DEV).long()

    def bounces(k):
        tri, st = _points(k, len(tris), gen)
        S, n = _surface(maps, wh, charts, tri, st)
        t1, t2 = _frame_of(n)
        u = torch.rand(k, 2, dtype=F8, device=DEV, generator=gen)
        r, phi = u[:, 0:1].sqrt(), 2.0 * math.pi * u[:, 1:2]
        d = r * phi.cos() * t1 + r * phi.sin() * t2 + (1.0 - u[:, 0:1]).sqrt() * n
        return S + 1e-4 * n, d, torch.full((k,), math.inf, dtype=F8, device=DEV)

    def grazing(k):
        tri, st = _points(k, len(tris), gen)
        g = {q: v[tri] for q, v in charts.items()}
        P, n = (g[a] + st[:, 0:1] * g[b] + st[:, 1:2] * g[c] for a, b, c in (("q0", "e1", "e2"), ("m0", "Mu", "Mv")))
        n = _unit(n)
        t1, t2 = _frame_of(n)
        u = torch.rand(k, 3, dtype=F8, device=DEV, generator=gen)
        phi = 2.0 * math.pi * u[:, 0:1]
        ang = torch.deg2rad(torch.exp(math.log(0.1) + u[:, 1:2] * math.log(50.0)))
        d = ang.cos() * (phi.cos() * t1 + phi.sin() * t2) - ang.sin() * n
        return P - (0.05 + 0.95 * u[:, 2:3]) * d, d, torch.full((k,), math.inf, dtype=F8, device=DEV)

    def shadows(k):
        tri, st = _points(k, len(tris), gen, 0.5)
        S, n = _surface(maps, wh, charts, tri, st)
        u = torch.rand(k, 2, dtype=F8, device=DEV, generator=gen)
        y = torch.stack([u[:, 0] * 0.5 - 0.25, torch.full_like(u[:, 0], 2.0), u[:, 1] * 0.5 - 0.25], 1)
        o = S + 1e-4 * n
        dist = (y - o).norm(dim=1)
        return o, (y - o) / dist[:, None], dist - 1e-4

    parts = {"camera": lambda: [_camera(case, m, gen)], "shadow": lambda: [shadows(m)],
             "frame": lambda: [_camera(case, m - m // 4, gen)] + ([bounces(m // 4)] if m >= 4 else []),
             "grazing": lambda: [_camera(case, m - m // 4 - m // 4, gen)] +
                                ([bounces(m // 4), grazing(m // 4)] if m >= 4 else [])}[mix]()
    out = torch.zeros(m, 8, dtype=torch.float32, device=DEV)
    out[:, 0:3], out[:, 3:6], out[:, 7] = (torch.cat(x).float() for x in zip(*parts))
    return out


# ---- states ----------------------------------------------------------------

def _options(case, **more):
    return dm.TraversalOptions(mode=case["mode"], order=case["order"], leaf_precision=case["leaf"],
                               graph=case["graph"], **more)


def _device_scene(maps, tris, which):
    ctx = context()
    assets = [dm.Asset(ctx, m.cpu().numpy()) for m in maps]
    return dm.Scene(ctx, assets, tris, which)


def _request_sizes(case):
    """Log-uniform request sizes (1 to 256) of the burst, and which are shadow-only."""
    rng = np.random.Generator(np.random.PCG64(case["requests"]))
    w = np.exp(rng.uniform(0.0, math.log(256.0), case["requests"]))
    n = np.maximum(1, (w / w.sum() * case["rays"]).astype(int))
    return n.tolist(), (rng.random(case["requests"]) < 0.1).tolist()


def prepare(case, seed):
    _forget()
    maps, (tris, which) = _maps(case, seed), _geometry(case)
    st = {"case": case}
    kind = case["kind"]
    if kind == "rebuild":
        st["nodes"] = maps[0].cpu().numpy()
        st["tris"], st["which"] = tris, which
    else:
        st["scene"] = _device_scene(maps, tris, which)
    if kind in ("query", "host", "rebuild"):
        rays = _rays(case, maps, tris, which, seed)
        st["options"] = _options(case)
        if kind == "host":
            st["rays"] = rays.cpu().numpy().astype(np.float64 if case["record"] == "f64" else np.float32)
        else:
            st["rays"] = rays.double() if case["record"] == "f64" else rays
            st["hits"] = torch.empty(case["rays"], 80 if case["record"] == "f64" else 48, dtype=torch.uint8,
                                     device=DEV)
    elif kind == "render":
        st["view"] = scenes.path_tracer_view(case["width"], case["height"])
        st["emitter"] = np.array([[-0.25, 2.0, -0.25], [0.25, 2.0, -0.25], [-0.25, 2.0, 0.25], [0.25, 2.0, 0.25]])
        st["seed"] = seed
    elif kind == "serve":
        sizes, shadow = _request_sizes(case)
        st["requests"] = [(_rays(case, maps, tris, which, seed + 31 * q, m).cpu().numpy(),
                           "occluded" if s else "closest") for q, (m, s) in enumerate(zip(sizes, shadow))]
        st["answers"] = [np.empty(m, dm.HIT32) for m in sizes]
        st["server"] = dm.Server(context(), max_batch_rays=1 << 20)
    elif kind == "mesh":
        n, t = case["sub"], len(tris)
        v, f = (n + 1) * (n + 2) // 2 * t, n * n * t
        st["mesh"] = [torch.empty(v, 3, device=DEV), torch.empty(v, 2, device=DEV), torch.empty(v, 3, device=DEV),
                      torch.empty(f, 3, dtype=torch.int32, device=DEV)]
    _forget()
    return st


def _answer(case, hits):
    """A device hit buffer as the values a caller reads: occlusion queries answer with the triangle alone."""
    width, real = (10, torch.float64) if case["record"] == "f64" else (12, torch.float32)
    ints = hits.view(torch.int32)[:, -4:]
    return {"tri": ints[:, 0:1]} if case["mode"] == "occluded" else {"hit": hits.view(real)[:, :8], "ids": ints}


def _host_answer(hits, mode):
    if mode == "occluded":
        return {"occluded": (hits["tri"] >= 0).astype(np.uint8)}
    real = np.float64 if hits.dtype == dm.HIT64 else np.float32
    flat = hits.view(np.uint8).reshape(len(hits), -1)
    return {"hit": np.ascontiguousarray(flat[:, :8 * np.dtype(real).itemsize]).view(real),
            "ids": np.ascontiguousarray(flat[:, -16:]).view(np.int32)}


def _query(case, scene, st):
    kind = dm.F64 if case["record"] == "f64" else dm.F32
    scene.intersect_device(st["rays"].data_ptr(), kind, case["rays"], st["hits"].data_ptr(), kind, st["options"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "query":
        _query(case, state["scene"], state)
        return _answer(case, state["hits"])
    if kind == "host":
        hits = state["scene"].intersect(state["rays"], state["options"], state["rays"].dtype)
        return _host_answer(hits, case["mode"])
    if kind == "rebuild":
        ctx = context()
        asset = dm.Asset(ctx, state["nodes"])
        scene = dm.Scene(ctx, [asset], state["tris"], state["which"])
        _query(case, scene, state)
        scene.close()
        asset.close()
        return _answer(case, state["hits"])
    if kind == "render":
        img, _, _ = state["scene"].render(state["view"], state["emitter"], spp=case["spp"], max_depth=5,
                                          seed=state["seed"])
        return img
    if kind == "serve":
        server = state["server"]
        for (rays, mode), hits in zip(state["requests"], state["answers"]):
            server.submit_rays(state["scene"], rays, mode, hits)
        server.drain()
        return [_host_answer(h, mode) for (_, mode), h in zip(state["requests"], state["answers"])]
    pos, tex, nrm, idx = state["mesh"]
    ctx = context()
    ctx.check(dm.lib().dmap_tessellate_uniform(state["scene"].h, case["sub"], ctypes.c_void_p(pos.data_ptr()),
                                               ctypes.c_void_p(tex.data_ptr()), ctypes.c_void_p(nrm.data_ptr()),
                                               ctypes.c_void_p(idx.data_ptr()), None), "dmap_tessellate_uniform")
    return [pos, tex, nrm, idx]


# ---- work --------------------------------------------------------------------

# The reference algorithm's work per ray, counted by the FP64 path on the
# benchmark's frame (62.9 node tests, 0.56 leaf tests, 13.4 sub-squares, 2.0
# Newton iterations; 450, 290, 285 and 215 operations each).
OPS_PER_RAY = 62.9 * 450 + 0.56 * 290 + 13.4 * 285 + 2.0 * 215


def work(case):
    kind, n, k = case["kind"], case["n"], case["k"]
    if kind == "mesh":
        t = 2 if case["scene"] == "quad" else 12 * k * k
        v, f = (case["sub"] + 1) * (case["sub"] + 2) // 2 * t, case["sub"] ** 2 * t
        return {"bytes": 32 * v + 12 * f, "flops": 250 * v}
    r = case["rays"]
    if kind == "render":
        # per sample one camera ray, about one bounce and one shadow ray a vertex; the image out
        return {"bytes": 12 * case["width"] * case["height"], "flops": 2 * r * OPS_PER_RAY}
    ray, hit = (64, 80) if case["record"] == "f64" else (32, 48)
    b = r * (ray + (4 if case["mode"] == "occluded" else hit))
    if kind == "rebuild":
        es = 2 if case["texel"] == "f16" else 4
        b += (n + 1) ** 2 * es + 32 * (4 * n * n // 3)
        return {"bytes": b, "flops": r * OPS_PER_RAY + 60 * n * n}
    return {"bytes": b, "flops": r * OPS_PER_RAY}


# ---- exact values -------------------------------------------------------------

class _Field:
    """A signed height above the displaced surface, f(x), whose zeros are the
    surface: on the quad z - h(x, y); on the sphere, whose base points equal
    its interpolated normals, so that a point's base point lies on the line
    to the centre, |x| - |P| - h(s, t)."""

    def __init__(self, case, maps, tris, which):
        self.case, self.maps = case, maps
        self.which = torch.from_numpy(which).to(DEV).long()
        self.charts = _charts(tris)
        self.quad = case["scene"] == "quad"
        if self.quad:
            return
        self.axes = torch.from_numpy(FACES).to(DEV)
        B = torch.stack([self.charts[q] for q in ("q0", "e1", "e2")], 2)  # x / l = q0 + s e1 + t e2
        self.inv = torch.linalg.inv(B)
        self.top = 1.0 + max(float(m.abs().max()) for m in maps)

    def at(self, x):
        """f, triangle and st of points x; triangle -1 outside the domain."""
        if self.quad:
            st = x[:, 0:2]
            tri = (st.sum(1) > 1.0).long()
            tri = torch.where(((st >= 0.0) & (st <= 1.0)).all(1), tri, -1)
            h, _ = _height(self.maps, torch.zeros_like(tri), st)
            return x[:, 2] - h, tri, st
        k = self.case["k"]
        face = (self.axes[:, 0] @ x.T).argmax(0)
        a = self.axes[face]
        w = (a[:, 0] * x).sum(1)
        c = torch.stack([(a[:, 1] * x).sum(1) / w, (a[:, 2] * x).sum(1) / w], 1)
        c = ((c + 1.0) * (0.5 * k)).clamp(0.0, k * (1.0 - 1e-15))
        cell = c.floor()
        patch = face * (k * k) + (cell[:, 1] * k + cell[:, 0]).long()
        tri = 2 * patch + ((c - cell).sum(1) > 1.0).long()
        q = (self.inv[tri] @ x[:, :, None])[..., 0]
        st = q[:, 1:3] / q[:, 0:1]
        base = x.norm(dim=1) / q[:, 0]
        h, _ = _height(self.maps, self.which[tri], st)
        return x.norm(dim=1) - base - h, tri, st

    def range(self, o, d):
        """The part of each ray that can meet the surface."""
        if self.quad:
            top = float(self.maps[0].abs().max()) * 1.001
            a, b = (-top - o[:, 2]) / d[:, 2], (top - o[:, 2]) / d[:, 2]
            return torch.minimum(a, b).clamp(min=0.0), torch.maximum(a, b).clamp(max=4.0)
        b, c = (o * d).sum(1) / (d * d).sum(1), ((o * o).sum(1) - self.top ** 2) / (d * d).sum(1)
        disc = b * b - c
        r = disc.clamp(min=0.0).sqrt()
        hi = torch.where(disc > 0.0, -b + r, torch.full_like(b, -1.0))
        return (-b - r).clamp(min=0.0), hi


def _first_root(F, o, d, a, fa, b, fb):
    """The first zero of f in [a, b] of each ray, where f changes sign there: (t, found)."""
    found = (fa > 0.0) != (fb > 0.0)
    lo, hi, flo = a.clone(), b.clone(), fa
    for _ in range(52):
        mid = 0.5 * (lo + hi)
        fm, _, _ = F.at(o + mid[:, None] * d)
        up = (fm > 0.0) == (flo > 0.0)
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    return 0.5 * (lo + hi), found


def _march(F, rays, texel):
    """The nearest crossing of each ray in (0, t_max). Steps of a quarter
    texel find where f changes sign, which ends the ray's march; on the way
    they note the steps that leave a patch (whose neighbour has another map)
    and the dips of f toward the surface, which are searched afterwards: the
    first by cutting the step at the patch's edge, the second for a pair of
    crossings around the dip's lowest point."""
    o, d = rays[:, 0:3].double(), rays[:, 3:6].double()
    a, b = F.range(o, d)
    b = torch.minimum(b, rays[:, 7].double())
    best = torch.full_like(a, math.inf)
    step = 0.25 * texel / d.norm(dim=1)
    idx = torch.nonzero(a < b)[:, 0]
    if not len(idx):
        return best

    def group(tri):
        return (tri >= 0).long() if F.quad else tri // 2

    def f_at(k, t):
        return F.at(o[k] + t[:, None] * d[k])

    def take(k, r, ok):
        r = torch.where(ok & (r > 0.0), r, math.inf)
        best.scatter_reduce_(0, k, r, "amin")

    t = a[idx]
    f, tri, _ = f_at(idx, t)
    t_old, f_old = t, f
    crossings, edges, dips = [], [], []
    while len(idx):
        t1 = torch.minimum(t + step[idx], b[idx])
        f1, tri1, _ = f_at(idx, t1)
        same = group(tri) == group(tri1)
        inside = same & (tri1 >= 0)
        cross = inside & ((f > 0.0) != (f1 > 0.0))
        dip = inside & ~cross & (f.abs() < f_old.abs()) & (f.abs() < f1.abs()) & (f.abs() < 0.5 * texel)
        for where, events in ((cross, crossings), (~same, edges), (dip, dips)):
            q = torch.nonzero(where)[:, 0]
            if len(q):
                events.append((idx[q], t_old[q], t[q], t1[q]))
        left = torch.nonzero(~cross & (t1 < b[idx]))[:, 0]
        new = ~same[left]  # a dip's search stays within one patch
        t_old, f_old = torch.where(new, t1[left], t[left]), torch.where(new, math.inf, f[left])
        idx, t, f, tri = idx[left], t1[left], f1[left], tri1[left]

    for k, _, x, y in [tuple(torch.cat(v) for v in zip(*crossings))] * bool(crossings):
        take(k, *_first_root(F, o[k], d[k], x, f_at(k, x)[0], y, f_at(k, y)[0]))
    for k, _, x, y in [tuple(torch.cat(v) for v in zip(*edges))] * bool(edges):
        lo, hi, first = x.clone(), y.clone(), group(f_at(k, x)[1])
        for _ in range(50):
            mid = 0.5 * (lo + hi)
            here = group(f_at(k, mid)[1]) == first
            lo, hi = torch.where(here, mid, lo), torch.where(here, hi, mid)
        for u, v in ((x, torch.maximum(lo - 1e-10, x)), (torch.minimum(hi + 1e-10, y), y)):  # clear of the edge
            (fu, _, _), (fv, tv, _) = f_at(k, u), f_at(k, v)
            r, ok = _first_root(F, o[k], d[k], u, fu, v, fv)
            take(k, r, ok & (tv >= 0) & (f_at(k, r)[1] >= 0))
    for k, x, m, y in [tuple(torch.cat(v) for v in zip(*dips))] * bool(dips):
        lo, hi, sign = x.clone(), y.clone(), torch.sign(f_at(k, m)[0])
        for _ in range(40):
            m1, m2 = lo + (hi - lo) / 3.0, hi - (hi - lo) / 3.0
            left = sign * f_at(k, m1)[0] < sign * f_at(k, m2)[0]
            lo, hi = torch.where(left, lo, m1), torch.where(left, m2, hi)
        m = 0.5 * (lo + hi)
        take(k, *_first_root(F, o[k], d[k], x, f_at(k, x)[0], m, f_at(k, m)[0]))
    return best


def _exact_hits(case, maps, tris, which, rays):
    """(m, 8) doubles t, st, bary, ng of the nearest crossings (misses: inf, zeros)."""
    F = _Field(case, maps, tris, which)
    texel = (1.0 if F.quad else 0.39 * 4.0 / case["k"]) / case["n"]
    t = _march(F, rays, texel)
    out = torch.zeros(len(rays), 8, dtype=F8, device=DEV)
    out[:, 0] = t
    hit = torch.nonzero(torch.isfinite(t))[:, 0]
    if len(hit):
        x = rays[hit, 0:3].double() + t[hit, None] * rays[hit, 3:6].double()
        _, tri, st = F.at(x)
        tri = tri.clamp(min=0)
        J, t0 = F.charts["J"][tri], F.charts["t0"][tri]
        out[hit, 1:3] = st
        out[hit, 3:5] = (J @ (st - t0)[:, :, None])[..., 0]
        out[hit, 5:8] = _surface(maps, F.which, F.charts, tri, st)[1]
    return out


def exact(case, seed):
    """Values from a march in 64 bits, for closest hits on the quad and the
    sphere while the rays times the steps they take stay within seconds, and
    for meshes. None for occlusion (whole numbers), larger batches, the path
    tracer's images and the server's bursts (more rays than that)."""
    kind = case["kind"]
    if kind in ("render", "serve") or case["mode"] == "occluded":
        return None
    steps = case["n"] * (6 if case["scene"] == "quad" else 30 * case["k"] / 4)
    if kind != "mesh" and (case["scene"] == "ground" or steps > 16000 or steps * case["rays"] > 2.0e9):
        return None
    _forget()
    maps, (tris, which) = _maps(case, seed), _geometry(case)
    if kind == "mesh":
        n = case["sub"]
        ij = torch.cat([torch.stack([torch.arange(n - j + 1, dtype=F8), torch.full((n - j + 1,), float(j),
                                                                                     dtype=F8)], 1)
                        for j in range(n + 1)]).to(DEV) / n
        T = torch.from_numpy(np.ascontiguousarray(tris)).to(DEV)[:, 18:24].view(-1, 1, 3, 2)
        st = T[:, :, 0] + ij[None, :, 0:1] * (T[:, :, 1] - T[:, :, 0]) + ij[None, :, 1:2] * (T[:, :, 2] - T[:, :, 0])
        tri = torch.arange(len(tris), device=DEV).repeat_interleave(len(ij))
        st = st.reshape(-1, 2)
        S, n_ = _surface(maps, torch.from_numpy(which).to(DEV).long(), _charts(tris), tri, st)
        _forget()
        return [S, st, n_, None]
    rays = _rays(case, maps, tris, which, seed)
    out = _exact_hits(case, maps, tris, which, rays)
    _forget()
    return {"hit": out.cpu().numpy() if kind == "host" else out, "ids": None}
