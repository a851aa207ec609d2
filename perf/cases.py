"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public Python entry points (Context.build / refit /
trace / trace_sorted / adjoint / primary_rays, Batch.build_trace). Five kinds:

  build   a mesh on the device becomes a BVH (rebuilt into a BVH object that the
          program keeps, as one does for geometry that changes every frame)
  trace   rays against a BVH that is already built: closest hits of incoherent
          rays, in their own or in Morton order, or the visibility of shadow rays
  camera  one frame of primary rays: generated on the device, then traced
  frame   build and trace of the same frame: geometry that changes every frame
  diff    one step of fitting a surface to measurements: refit to the current
          vertices, trace, gradient of a loss over (t, u, v)
  batch   many meshes of uneven size built and traced by one captured graph

Meshes: "soup" is a uniform triangle soup, "clusters" triangles of Gaussian
clusters, "mixed" the two interleaved (all three with vertices of their own per
triangle), "terrain" an indexed heightfield.
"""
import math

import numpy as np
import torch

import hippie_b200 as hp

# A ray's largest distance: beyond every scene here (all lie about [0, 1]^3 and
# rays start at most 1.5 from a face), and finite so that misses have a value.
FAR = 4.0


def listed():
    return [
        # The smallest rebuild: one prop of an editor's or game's scene. Latency.
        {"name": "build_lbvh_5k", "kind": "build", "method": "lbvh", "bits": 30, "mesh": "soup", "n": 5003,
         "layout": 2},
        # An ordinary object rebuilt with the better tree, at an odd size.
        {"name": "build_ploc_100k", "kind": "build", "method": "ploc", "bits": 60, "mesh": "clusters", "n": 100003,
         "layout": 2},
        # The headline build: a whole scene by PLOC (radius 16, 60-bit keys).
        {"name": "build_ploc_4m", "kind": "build", "method": "ploc", "bits": 60, "mesh": "clusters", "n": 4194304,
         "layout": 2},
        # The largest build: a scan-sized mesh by the fastest builder.
        {"name": "build_lbvh_16m", "kind": "build", "method": "lbvh", "bits": 60, "mesh": "mixed", "n": 16777259,
         "layout": 2},
        # A static scene's tree, worth restructuring (treelets of 9, 2 rounds).
        {"name": "build_atr_1m", "kind": "build", "method": "atr", "bits": 60, "mesh": "clusters", "n": 1048573,
         "layout": 2},
        # A frame of a dynamic scene in the four-wide layout: build, then closest hits.
        {"name": "frame_quad_500k", "kind": "frame", "method": "ploc", "bits": 60, "mesh": "clusters", "n": 500009,
         "layout": 4, "rays": 1000003},
        # The headline trace: incoherent (diffuse bounce) rays in a whole scene.
        {"name": "trace_bounce_16m", "kind": "trace", "method": "ploc", "bits": 60, "mesh": "clusters", "n": 4194304,
         "layout": 2, "rays": 16777216, "mode": "closest"},
        # A frame's primary rays at 1080p over a terrain (coherent).
        {"name": "camera_1080p", "kind": "camera", "method": "lbvh", "bits": 60, "mesh": "terrain", "nx": 512,
         "ny": 512, "layout": 2, "w": 1920, "h": 1080},
        # Shadow rays of a frame: visibility only, on a small scene.
        {"name": "trace_shadow_1m", "kind": "trace", "method": "lbvh", "bits": 30, "mesh": "soup", "n": 65536,
         "layout": 2, "rays": 1048576, "mode": "any"},
        # Bounce rays that the tracer is asked to order first, at odd sizes.
        {"name": "trace_sorted_4m", "kind": "trace", "method": "lbvh", "bits": 60, "mesh": "mixed", "n": 1000003,
         "layout": 2, "rays": 4000037, "mode": "sorted"},
        # Fitting a 512 x 1024 heightfield: forward, backward, refit.
        {"name": "diff_terrain_4m", "kind": "diff", "nx": 512, "ny": 1024, "rx": 2048, "ry": 2048},
        # 256 meshes, log-uniform in size, four rays a triangle.
        {"name": "batch_256", "kind": "batch", "bits": 30, "meshes": 256, "lo": 256, "hi": 262144},
    ]


def _log(rng, lo, hi):
    """A size drawn uniformly over the logarithm, odd more often than not."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, v | 1) if rng.random() < 0.7 else v


def _draw_mesh(rng, lo, hi):
    mesh = rng.choice(["soup", "clusters", "mixed", "terrain"])
    if mesh != "terrain":
        return {"mesh": mesh, "n": _log(rng, lo, hi)}
    n = _log(rng, lo, hi)
    nx = max(2, int(math.sqrt(n / 2) * math.exp(rng.uniform(-0.5, 0.5))))
    return {"mesh": mesh, "nx": nx, "ny": max(2, min(n // (2 * nx), hi // (2 * nx)))}


def draw(rng):
    kind = rng.choice(["build", "build", "trace", "trace", "camera", "frame", "diff", "batch"])
    method = rng.choice(["lbvh", "ploc", "atr", "hlbvh"])
    bits = rng.choice([30, 60])
    layout = rng.choice([2, 2, 2, 4, 8])
    if kind == "build":
        big = {"lbvh": 12000000, "ploc": 4000000, "atr": 2000000, "hlbvh": 4000000}[method]
        return {"kind": kind, "method": method, "bits": bits, "layout": layout, **_draw_mesh(rng, 4000, big)}
    if kind == "trace":
        return {"kind": kind, "method": method, "bits": bits, "layout": layout, **_draw_mesh(rng, 4000, 2000000),
                "rays": _log(rng, 60000, 8000000), "mode": rng.choice(["closest", "any", "sorted"])}
    if kind == "camera":
        w = _log(rng, 300, 2600)
        return {"kind": kind, "method": method, "bits": bits, "layout": layout, **_draw_mesh(rng, 4000, 2000000),
                "w": w, "h": max(1, w * 9 // 16)}
    if kind == "frame":
        return {"kind": kind, "method": method, "bits": bits, "layout": layout, **_draw_mesh(rng, 4000, 1000000),
                "rays": _log(rng, 60000, 4000000)}
    if kind == "diff":
        return {"kind": kind, "nx": _log(rng, 40, 700), "ny": _log(rng, 40, 700), "rx": _log(rng, 200, 2000),
                "ry": _log(rng, 200, 2000)}
    return {"kind": kind, "bits": min(bits, 48), "meshes": _log(rng, 16, 256), "lo": 256, "hi": _log(rng, 4096, 131072)}


# ---- inputs, made on the GPU from the seed --------------------------------------
def _gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + what) & 0x7fffffff)
    return g


def _u(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _centres(g, mesh, n):
    if mesh == "soup":
        return _u(g, n, 3)
    c = _u(g, 1024, 3)
    return c[torch.arange(n, device="cuda") % 1024] + 0.02 * torch.randn(n, 3, generator=g, device="cuda")


def _terrain(g, nx, ny, sy=1.0):
    """z = a sum of 16 sinusoids over [0, 1] x [0, sy]; two triangles a cell."""
    y, x = torch.meshgrid(torch.linspace(0, sy, ny, device="cuda", dtype=torch.float64),
                          torch.linspace(0, 1, nx, device="cuda", dtype=torch.float64), indexing="ij")
    k = torch.rand(16, 4, generator=g, device="cuda", dtype=torch.float64)
    z = torch.zeros_like(x)
    for a, f, th, ph in k.tolist():
        f = 2 * math.pi * (1 + 31 * f)
        z += 0.05 * a * torch.sin(f * (math.cos(2 * math.pi * th) * x + math.sin(2 * math.pi * th) * y)
                                  + 2 * math.pi * ph)
    v = torch.stack([x, y, z], -1).reshape(-1, 3).float().contiguous()
    a = (torch.arange(ny - 1, device="cuda")[:, None] * nx + torch.arange(nx - 1, device="cuda")[None]).reshape(-1)
    t = torch.stack([a, a + 1, a + nx + 1, a, a + nx + 1, a + nx], -1).reshape(-1, 3)
    return v, t.int().contiguous()


def _mesh(case, seed, what=1):
    g = _gen(seed, what)
    if case["mesh"] == "terrain":
        return _terrain(g, case["nx"], case["ny"])
    n = case["n"]
    if case["mesh"] == "mixed":
        c = torch.empty(n, 3, device="cuda")
        c[0::2] = _centres(g, "soup", (n + 1) // 2)
        c[1::2] = _centres(g, "clusters", n // 2)
    else:
        c = _centres(g, case["mesh"], n)
    h = 0.005 if case["mesh"] == "clusters" else 0.01
    v = c[:, None, :] + (2 * _u(g, n, 3, 3) - 1) * h
    return v.reshape(-1, 3).contiguous(), torch.arange(3 * n, device="cuda", dtype=torch.int32).reshape(n, 3)


def _sphere_rays(g, n, v):
    """Origins uniform in the mesh's box, directions uniform on the sphere."""
    lo, hi = v.amin(0), v.amax(0)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float32)
    r = torch.empty(n, 8, device="cuda")
    r[:, :3] = lo + (hi - lo) * _u(g, n, 3)
    r[:, 3] = 0
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True).clamp_min(1e-20)
    r[:, 7] = FAR
    return r


def _shadow_rays(g, n, v):
    """From points in the mesh's box towards points of a light above it."""
    lo, hi = v.amin(0), v.amax(0)
    o = lo + (hi - lo) * _u(g, n, 3)
    light = torch.cat([lo[:2] + (hi - lo)[:2] * (0.3 + 0.4 * _u(g, n, 2)), (hi[2] + 0.5).expand(n, 1)], 1)
    d = light - o
    r = torch.empty(n, 8, device="cuda")
    r[:, :3] = o
    r[:, 3] = 1e-4
    r[:, 7] = d.norm(dim=1)
    r[:, 4:7] = d / r[:, 7:8]
    return r


def _trace_rays(case, seed, v):
    g = _gen(seed, 2)
    return (_shadow_rays if case.get("mode") == "any" else _sphere_rays)(g, case["rays"], v)


def _grid_rays(case, seed):
    """Downward rays, one in each cell of an rx x ry grid over [0, 1] x [0, 2]."""
    g = _gen(seed, 2)
    rx, ry = case["rx"], case["ry"]
    j, i = torch.meshgrid(torch.arange(ry, device="cuda"), torch.arange(rx, device="cuda"), indexing="ij")
    r = torch.zeros(rx * ry, 8, device="cuda")
    r[:, 0] = (i.reshape(-1) + _u(g, rx * ry)) / rx
    r[:, 1] = (j.reshape(-1) + _u(g, rx * ry)) * 2 / ry
    r[:, 2] = 1
    r[:, 6] = -1
    r[:, 7] = 2
    return r


def _sizes(case):
    """Triangles of the batch's meshes: log-uniform, the same for every seed (a
    batch's sizes are part of the case)."""
    rng = np.random.default_rng(case["meshes"] * 1000003 + case["hi"])
    return np.round(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["meshes"]))).astype(np.int64)


# ---- state ----------------------------------------------------------------------
_CTX = _STREAM = None


def _ctx():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = hp.Context(0)
    return _CTX


def _stream():
    """The one stream on which the program launches its batches (a captured graph
    needs one that is not the default; calls of one context follow one another)."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _params(case):
    kw = dict(method=case["method"], morton_bits=case["bits"], layout=case.get("layout", 2))
    if case["method"] == "ploc":
        kw.update(ploc_radius=16, ploc_max_radius=256)
    if case["method"] == "atr":
        kw.update(atr_treelet=9, atr_iterations=2)
    if case["method"] == "hlbvh":
        kw.update(hlbvh_sah_bits=15)
    return hp.BuildParams(**kw)


def _bvh(ctx, n, layout=2):
    """Storage for a BVH of n triangles and its device arrays, zero where no build
    has written. They are views of the BVH's own memory, so each keeps it alive."""
    bvh = hp.BVH.reserve(ctx, n, layout)
    out = dict(zip(("nodes", "woop", "index"), bvh.arrays()))
    for x in out.values():
        x.zero_()
        x.owner = bvh
    return bvh, out


def _results(n):
    res = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    return res, {"tri": res[:, 0], "tuv": res.view(torch.float32)[:, 1:]}


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        sizes = _sizes(case)
        at = np.concatenate([[0], np.cumsum(sizes)]).tolist()
        v, _ = _mesh({"mesh": "soup", "n": at[-1]}, seed)
        t = torch.arange(3 * int(sizes.max()), device="cuda", dtype=torch.int32).reshape(-1, 3)
        s["meshes"] = [(v[3 * at[i]:3 * at[i + 1]], t[:at[i + 1] - at[i]]) for i in range(len(sizes))]
        s["stream"] = _stream()
        s["batch"] = hp.Batch(ctx, s["meshes"], [int(4 * k) for k in sizes],
                              hp.BuildParams(method="lbvh", morton_bits=case["bits"]))
        s["rays"] = _sphere_rays(_gen(seed, 2), s["batch"].num_rays, v)
        s["res"], s["out"] = _results(s["batch"].num_rays)
        torch.cuda.synchronize()
        return s
    if kind == "diff":
        # The BVH was built on the vertices the fit began with; the current ones
        # have moved since.
        v0, s["t"] = _terrain(_gen(seed, 1), case["nx"], case["ny"], 2.0)
        s["bvh"], tree = _bvh(ctx, s["t"].shape[0])
        ctx.build(v0, s["t"], hp.BuildParams(method="lbvh", morton_bits=60), bvh=s["bvh"])
        s["v"] = _moved(case, seed, v0)
        s["rays"] = _grid_rays(case, seed)
        s["w"] = torch.randn(s["rays"].shape[0], 3, generator=_gen(seed, 4), device="cuda")
        s["grad"] = torch.zeros_like(s["v"])
        s["res"], s["out"] = _results(s["rays"].shape[0])
        s["out"] = {**s["out"], "grad": s["grad"], **tree}
        return s
    s["v"], s["t"] = _mesh(case, seed)
    s["params"] = _params(case)
    s["bvh"], tree = _bvh(ctx, s["t"].shape[0], case["layout"])
    s["out"] = tree if kind in ("build", "frame") else {}
    if not s["out"]:
        ctx.build(s["v"], s["t"], s["params"], bvh=s["bvh"])
    if kind == "camera":
        w, h = case["w"], case["h"]
        side = 0.4 * (torch.rand(2, generator=torch.Generator().manual_seed(int(seed) & 0x7fffffff)) - 0.5)
        pos = np.array([0.5 + float(side[0]), -0.9, 0.9 + float(side[1])], np.float32)
        look = np.array([0.5, 0.5, 0.0], np.float32) - pos
        s["pos"] = pos
        s["cam"] = hp.camera_screen_to_world(pos, look / np.linalg.norm(look), 45.0, w, h, 0.01, 100.0)
        s["wh"] = (w, h)
        s["table"] = torch.from_numpy(hp.pixel_table(w, h)).cuda()
        s["rays"] = torch.zeros(w * h, 8, device="cuda")
        s["out"]["rays"] = s["rays"]
    else:
        s["rays"] = _trace_rays(case, seed, s["v"]) if "rays" in case else None
        s["mode"] = case.get("mode", "closest")
    if s["rays"] is not None:
        s["res"], out = _results(s["rays"].shape[0])
        s["out"].update(out)
    return s


def _moved(case, seed, v):
    """The fit's current vertices: heights moved by up to a cell's size."""
    d = torch.zeros_like(v)
    d[:, 2] = (2 * _u(_gen(seed, 3), v.shape[0]) - 1) * (0.2 / max(case["nx"], case["ny"]))
    return (v + d).contiguous()


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "batch":
        s["batch"].build_trace(s["rays"], results=s["res"], stream=s["stream"])
    elif kind == "diff":
        ctx.refit(s["bvh"], s["v"], s["t"])
        ctx.trace(s["bvh"], s["rays"], results=s["res"])
        s["grad"].zero_()
        ctx.adjoint(s["v"], s["t"], s["rays"], s["res"], s["w"], dl_dverts=s["grad"])
    elif kind == "build":
        ctx.build(s["v"], s["t"], s["params"], bvh=s["bvh"])
    elif kind == "frame":
        ctx.build(s["v"], s["t"], s["params"], bvh=s["bvh"])
        ctx.trace(s["bvh"], s["rays"], results=s["res"])
    elif kind == "camera":
        ctx.primary_rays(s["pos"], s["cam"], *s["wh"], max_dist=FAR, index_to_pixel=s["table"], out=s["rays"])
        ctx.trace(s["bvh"], s["rays"], results=s["res"])
    elif s["mode"] == "any":
        # A shadow pass uses only whether something lies between.
        ctx.trace(s["bvh"], s["rays"], results=s["res"], any_hit=True)
        return {"lit": s["res"][:, 0] < 0}
    elif s["mode"] == "sorted":
        ctx.trace_sorted(s["bvh"], s["rays"], results=s["res"])
    else:
        ctx.trace(s["bvh"], s["rays"], results=s["res"])
    return s["out"]


# ---- what a pass cannot do without, and how exact it is -----------------------------
def _counts(case):
    """Vertices and triangles."""
    if "nx" in case:
        return case["nx"] * case["ny"], 2 * (case["nx"] - 1) * (case["ny"] - 1)
    return 3 * case["n"], case["n"]


def _trace_work(n, rays):
    """Rays read, hits written, the BVH (a 64-byte node and three 16-byte rows a
    triangle) read once; a ray tests two boxes of 15 operations on the way down
    to one triangle of 40."""
    return 48 * rays + 112 * n, rays * (30 * max(1.0, math.log2(max(n, 2))) + 40)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = int(_sizes(case).sum())
        b, f = _trace_work(n, 4 * n)
        return {"bytes": b + 48 * n + 116 * n, "flops": f + 150 * n}
    nv, n = _counts(case)
    mesh = 12 * nv + 12 * n
    # a 64-byte node, 48 bytes of intersection rows and an index a triangle; about
    # 150 operations for its box, code and rows
    build_b, build_f = mesh + 116 * n, 150 * n
    rays = case["rx"] * case["ry"] if kind == "diff" else case["w"] * case["h"] if kind == "camera" else \
        case.get("rays", 0)
    b, f = _trace_work(n, rays)
    if kind == "build":
        return {"bytes": build_b, "flops": build_f}
    if kind == "frame":
        return {"bytes": build_b + b, "flops": build_f + f}
    if kind == "diff":  # loss weights and directions read, the gradient written; the refit writes boxes and rows
        return {"bytes": build_b + b + 12 * rays + 12 * nv, "flops": build_f + f + 120 * rays}
    if kind == "camera":  # the pixel table read, the rays written
        return {"bytes": b + 36 * rays, "flops": f + 50 * rays}
    return {"bytes": b, "flops": f}


def tolerance(case):
    # Trees are integers, and boxes are copies of input values; hits are decided
    # and computed by one fixed sequence of roundings, with ties by triangle
    # number. Only the gradient is a 32-bit sum whose order is open.
    return {"rel": 1e-5} if case["kind"] == "diff" else "exact"


# ---- the same in 64 bits ------------------------------------------------------------
def _rows64(v, t):
    """Per triangle the affine map to (u, v, height), 3 x 4, in 64 bits."""
    p = v.double()[t.long()]
    a, b, c = p[:, 0] - p[:, 2], p[:, 1] - p[:, 2], p[:, 2]
    m = torch.stack([a, b, torch.linalg.cross(a, b)], -1)
    inv = torch.linalg.inv(m)
    return torch.cat([inv, -(inv @ c[:, :, None])], -1)


def _brute64(v, t, rays, tmin):
    """Closest hits by testing every triangle: (t, u, v), t = FAR without a hit."""
    w = _rows64(v, t)
    n, m = t.shape[0], rays.shape[0]
    out = torch.zeros(m, 3, dtype=torch.float64, device="cuda")
    step = max(1, 120000000 // max(n, 1))
    for i in range(0, m, step):
        r = rays[i:i + step].double()
        o = torch.cat([r[:, :3], torch.ones_like(r[:, :1])], 1)
        oz, dz = o @ w[:, 2].T, r[:, 4:7] @ w[:, 2, :3].T
        tt = -oz / dz
        u = o @ w[:, 0].T + tt * (r[:, 4:7] @ w[:, 0, :3].T)
        vv = o @ w[:, 1].T + tt * (r[:, 4:7] @ w[:, 1, :3].T)
        ok = (tt > tmin) & (tt < r[:, 7:8]) & (u >= 0) & (vv >= 0) & (u + vv <= 1)
        best, at = torch.where(ok, tt, math.inf).min(1)
        hit = torch.isfinite(best)
        k = torch.arange(r.shape[0], device="cuda")
        out[i:i + step, 0] = torch.where(hit, best, r[:, 7])
        out[i:i + step, 1] = torch.where(hit, u[k, at], 0.0)
        out[i:i + step, 2] = torch.where(hit, vv[k, at], 0.0)
    return out


def _terrain_hits64(v, nx, ny, rays):
    """The triangle under each downward ray, by its grid cell: (triangle, t, u, v)."""
    v = v.double().reshape(ny, nx, 3)
    x, y = rays[:, 0].double().contiguous(), rays[:, 1].double().contiguous()
    i = (torch.searchsorted(v[0, :, 0].contiguous(), x, right=True) - 1).clamp(0, nx - 2)
    j = (torch.searchsorted(v[:, 0, 1].contiguous(), y, right=True) - 1).clamp(0, ny - 2)
    fx = (x - v[j, i, 0]) / (v[j, i + 1, 0] - v[j, i, 0])
    fy = (y - v[j, i, 1]) / (v[j + 1, i, 1] - v[j, i, 1])
    return 2 * (j * (nx - 1) + i) + (fy > fx).long()


def exact(case, seed):
    kind = case["kind"]
    none = {"tri": None, "tuv": None}
    if kind == "build":
        return None  # a tree: numbers of nodes and triangles, and copies of the input's coordinates
    if kind == "diff":
        v0, t = _terrain(_gen(seed, 1), case["nx"], case["ny"], 2.0)
        vert = _moved(case, seed, v0).double().requires_grad_(True)
        rays = _grid_rays(case, seed)
        tri = _terrain_hits64(vert.detach(), case["nx"], case["ny"], rays)
        p = vert[t.long()[tri]]
        o, d = rays[:, :3].double(), rays[:, 4:7].double()
        a, b = p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]
        nrm = torch.linalg.cross(a, b)
        tt = ((p[:, 2] - o) * nrm).sum(1) / (d * nrm).sum(1)
        q = o + tt[:, None] * d - p[:, 2]
        nn = (nrm * nrm).sum(1)
        u = (torch.linalg.cross(q, b) * nrm).sum(1) / nn
        vv = (torch.linalg.cross(a, q) * nrm).sum(1) / nn
        tuv = torch.stack([tt, u, vv], 1)
        w = torch.randn(rays.shape[0], 3, generator=_gen(seed, 4), device="cuda").double()
        (tuv * w).sum().backward()
        return {**none, "tuv": tuv.detach(), "grad": vert.grad, "nodes": None, "woop": None, "index": None}
    if kind == "batch":
        sizes = _sizes(case)
        if int((4 * sizes * sizes).sum()) > 60e9:
            return None
        v, t = _mesh({"mesh": "soup", "n": int(sizes.sum())}, seed)
        rays = _sphere_rays(_gen(seed, 2), 4 * int(sizes.sum()), v)
        at = np.concatenate([[0], np.cumsum(sizes)]).tolist()
        return {**none, "tuv": torch.cat([_brute64(v, t[at[i]:at[i + 1]], rays[4 * at[i]:4 * at[i + 1]], 0.0)
                                          for i in range(len(sizes))])}
    nv, n = _counts(case)
    if kind == "camera" or case.get("mode") == "any" or n * case["rays"] > 60e9:
        return None
    v, t = _mesh(case, seed)
    tuv = _brute64(v, t, _trace_rays(case, seed, v), 0.0)
    return {**none, "tuv": tuv, **({"nodes": None, "woop": None, "index": None} if kind == "frame" else {})}
