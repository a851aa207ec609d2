"""Closest-hit adjoint and refit-only update on a heightfield (sm_100a).

The adjoint is checked against the FP64 closed-form gradient (oracle) and
against FP64 central finite differences; the refit against boxes recomputed
from the moved vertices over the same topology.
"""
import numpy as np
import pytest
import torch

import hippie_b200 as hp
import oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _scene(nx=64, ny=128, rx=256, ry=512, seed=3):
    v, t = hp.gen.heightfield(seed, nx, ny)
    rays = hp.gen.rays_grid_down(seed + 1, rx, ry)
    return v, t, rays


def test_adjoint_vs_fp64(ctx):
    v, t, rays = _scene()
    V, T, R = dev(v), dev(t), dev(rays)
    bvh = ctx.build(V, T, hp.BuildParams(morton_bits=60))
    res = ctx.trace(bvh, R)
    rng = np.random.default_rng(0)
    dl = rng.standard_normal((rays.shape[0], 3)).astype(np.float32)
    g = ctx.adjoint(V, T, R, res, dev(dl)).cpu().numpy().astype(np.float64)
    ctx.check()
    res_np = res.cpu().numpy()
    assert (res_np[:, 0] >= 0).mean() > 0.99
    ref = oracle.adjoint64(v, t, rays, res_np, dl)
    scale = np.abs(ref).max()
    err = np.abs(g - ref)
    assert err.max() <= 1e-3 * scale
    rel = np.linalg.norm(g - ref) / np.linalg.norm(ref)
    assert rel < 1e-4


def test_adjoint_vs_finite_differences(ctx):
    v, t, rays = _scene(nx=32, ny=64, rx=128, ry=256, seed=7)
    V, T, R = dev(v), dev(t), dev(rays)
    bvh = ctx.build(V, T, hp.BuildParams(morton_bits=60))
    res = ctx.trace(bvh, R).cpu().numpy()
    rng = np.random.default_rng(1)
    dl = rng.standard_normal((rays.shape[0], 3)).astype(np.float32)
    g = ctx.adjoint(V, T, R, dev(res), dev(dl)).cpu().numpy().astype(np.float64)
    hit = res[:, 0]
    # rays per triangle
    by_tri = {}
    for r in np.nonzero(hit >= 0)[0]:
        by_tri.setdefault(int(hit[r]), []).append(int(r))
    tri_of_vertex = {}
    for ti, tri in enumerate(t):
        for k in tri:
            tri_of_vertex.setdefault(int(k), []).append(ti)
    h = 1e-5
    an_all, fd_all = [], []
    interior = [i for i in range(v.shape[0]) if 0 < i % 32 < 31 and 0 < i // 32 < 63]
    for vid in rng.choice(interior, 200, replace=False):
        rs = [(r, ti) for ti in tri_of_vertex[int(vid)] for r in by_tri.get(ti, [])]
        if not rs:
            continue
        for axis in range(3):
            fd = 0.0
            stable = True
            for sgn in (+1, -1):
                vv = v.astype(np.float64).copy()
                vv[vid, axis] += sgn * h
                loss = 0.0
                for r, ti in rs:
                    p = vv[t[ti]]
                    ok, tuv = oracle.intersect64(p[0], p[1], p[2], rays[r, :3].astype(np.float64),
                                                 rays[r, 4:7].astype(np.float64))
                    if not ok:
                        stable = False
                        break
                    loss += dl[r, 0] * tuv[0] + dl[r, 1] * tuv[1] + dl[r, 2] * tuv[2]
                if not stable:
                    break
                fd += sgn * loss
            if not stable:
                continue
            fd /= 2 * h
            an_all.append(g[vid, axis])
            fd_all.append(fd)
        if len(fd_all) >= 512:
            break
    an_all, fd_all = np.array(an_all), np.array(fd_all)
    assert fd_all.size >= 100
    # Tolerance: 1e-3 relative, norm-wise over the sampled coordinates; per
    # coordinate 1e-3 relative plus 1e-4 of the largest sampled gradient, since a
    # vertex gradient is a sum of per-ray terms that can cancel to far below them.
    rel = np.linalg.norm(an_all - fd_all) / np.linalg.norm(fd_all)
    assert rel <= 1e-3, rel
    bound = 1e-3 * np.abs(fd_all) + 1e-4 * np.abs(fd_all).max()
    bad = np.abs(an_all - fd_all) > bound
    assert not bad.any(), list(zip(an_all[bad], fd_all[bad]))


def test_refit_after_vertex_step(ctx):
    v, t, rays = _scene(nx=64, ny=128, rx=128, ry=256, seed=11)
    V, T, R = dev(v), dev(t), dev(rays)
    bvh = ctx.build(V, T, hp.BuildParams(morton_bits=60))
    before = bvh.download()[0]
    rng = np.random.default_rng(5)
    v2 = v.copy()
    v2[:, 2] += rng.uniform(-0.01, 0.01, v.shape[0]).astype(np.float32)
    V2 = dev(v2)
    ctx.refit(bvh, V2, T)
    ctx.check()
    nodes, woop, tri = bvh.download()
    # topology unchanged
    np.testing.assert_array_equal(nodes[:, 12:], before[:, 12:])
    # woop equals a fresh woopify of the moved triangles
    ref_woop = np.zeros_like(woop)
    oracle.load().or_woopify(tri.shape[0], v2.ctypes.data, t.ctypes.data, tri.ctypes.data, ref_woop.ctypes.data)
    np.testing.assert_array_equal(woop.view(np.int32), ref_woop.view(np.int32))
    # every node's child boxes are the exact boxes of the moved geometry below them
    n_int = bvh.c.num_interior
    f = nodes[:, :12].view(np.float32)

    def node_box(i):
        if nodes[i, 14] < 0:
            b, e = nodes[i, 12], nodes[i, 13]
            p = v2[t[tri[b:e]]].reshape(-1, 3)
            return p.min(0), p.max(0)
        (a0, a1), (b0, b1) = node_box(child(i, 0)), node_box(child(i, 1))
        return np.minimum(a0, b0), np.maximum(a1, b1)

    def child(i, k):
        c = nodes[i, 12 + k]
        return ~c if c < 0 else c

    import sys
    sys.setrecursionlimit(10000)
    for i in rng.choice(n_int, 200, replace=False):
        for k in range(2):
            mn, mx = node_box(child(i, k))
            got_mn = np.array([f[i, 4 * k + 0], f[i, 4 * k + 2], f[i, 8 + 2 * k]])
            got_mx = np.array([f[i, 4 * k + 1], f[i, 4 * k + 3], f[i, 9 + 2 * k]])
            np.testing.assert_array_equal(got_mn, mn)
            np.testing.assert_array_equal(got_mx, mx)
    assert bvh.validate(V2, T)
    # tracing the refitted BVH equals the oracle on the refitted data
    got = ctx.trace(bvh, R, results=torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda"))
    np.testing.assert_array_equal(got.cpu().numpy(), oracle.trace(nodes, woop, tri, rays))


class _ClosestHitTUV(torch.autograd.Function):
    """(t, u, v) of each ray's closest hit as a differentiable function of the
    vertices (misses give zeros); backward is the library's adjoint kernel."""

    @staticmethod
    def forward(fctx, V, T, R, bvh, hctx):
        res = hctx.trace(bvh, R, results=torch.zeros((R.shape[0], 4), dtype=torch.int32, device=R.device))
        fctx.save_for_backward(V, T, R, res)
        fctx.hctx = hctx
        tuv = res[:, 1:].view(torch.float32).clone()
        tuv[res[:, 0] < 0] = 0.0
        return tuv

    @staticmethod
    def backward(fctx, g):
        V, T, R, res = fctx.saved_tensors
        gv = fctx.hctx.adjoint(V, T, R, res, g.contiguous())
        return gv, None, None, None, None


def test_autograd_function_gradient_and_refit_step(ctx):
    v, t, rays = _scene(nx=48, ny=96, rx=192, ry=384, seed=13)
    V, T, R = dev(v), dev(t), dev(rays)
    V.requires_grad_(True)
    p = hp.BuildParams(morton_bits=60)
    bvh = ctx.build(V.detach(), T, p)
    w = dev(np.random.default_rng(2).standard_normal((rays.shape[0], 3)).astype(np.float32))
    tuv = _ClosestHitTUV.apply(V, T, R, bvh, ctx)
    loss = (w * tuv).sum()
    loss.backward()
    ctx.check()
    res = ctx.trace(bvh, R).cpu().numpy()
    ref = oracle.adjoint64(v, t, rays, res, w.cpu().numpy())  # FP64 reference gradient
    g = V.grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - ref) / np.linalg.norm(ref) < 1e-4
    # one gradient step on z, refit, and trace again: same hits as a fresh build
    with torch.no_grad():
        V2 = V.detach().clone()
        V2[:, 2] -= 1e-4 * V.grad[:, 2] / V.grad[:, 2].abs().max()
    ctx.refit(bvh, V2, T)
    fresh = ctx.build(V2, T, p)
    a = ctx.trace(bvh, R, results=torch.zeros((R.shape[0], 4), dtype=torch.int32, device="cuda")).cpu().numpy()
    b = ctx.trace(fresh, R, results=torch.zeros((R.shape[0], 4), dtype=torch.int32, device="cuda")).cpu().numpy()
    # the closest hit does not depend on the tree (ties go to the lower id) except
    # where a slab test rounds a node away; allow that on a handful of rays
    assert np.mean(np.all(a == b, axis=1)) > 0.9999


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("group", [1, 3, 32, 77])
def test_adjoint_groups_and_alignment(ctx, group, shift):
    """Runs of `group` rays on one triangle (lanes of a warp that sum before they add:
    one, a few, a whole warp, runs across warps) and every third ray on another
    triangle between them, with all buffers 0 or 4 bytes past an 8-byte boundary."""
    n = 4099

    def at(a):  # the array, `shift` words into a buffer
        x = torch.from_numpy(np.ascontiguousarray(a)).reshape(-1)
        buf = torch.zeros(x.numel() + shift, dtype=x.dtype, device="cuda")
        buf[shift:] = x.cuda()
        return buf[shift:].reshape(a.shape)

    v, t, _ = _scene(17, 19)
    v[:, 2] *= 0.1  # gentle slopes: no triangle near edge-on, whose determinant cancels
    rng = np.random.default_rng(group)
    tri = (np.arange(n) // group) % len(t)
    tri[::3] = (tri[::3] * 7 + 3) % len(t)
    # a ray through a chosen point of its triangle, one unit before it (the oracle
    # takes the barycentrics from the ray)
    uv = rng.uniform(0.1, 0.45, (n, 2))
    p = v[t[tri]].astype(np.float64)
    at_p = uv[:, :1] * p[:, 0] + uv[:, 1:] * p[:, 1] + (1 - uv.sum(1, keepdims=True)) * p[:, 2]
    rays = np.zeros((n, 8), np.float32)
    rays[:, 4:7] = rng.normal(size=(n, 3)) * 0.1 + [0, 0, -1]
    rays[:, :3] = at_p - rays[:, 4:7]
    res = np.zeros((n, 4), np.int32)
    res[:, 0] = np.where(rng.random(n) < 0.05, -1, tri)
    res[:, 1] = np.ones(n, np.float32).view(np.int32)
    res[:, 2:] = uv.astype(np.float32).view(np.int32)
    w = rng.standard_normal((n, 3)).astype(np.float32)
    grad = at(np.zeros_like(v))
    # rays and results keep the 16-byte alignment of their records
    ctx.adjoint(at(v), at(t), dev(rays), dev(res), at(w), dl_dverts=grad)
    ctx.check()
    exp = oracle.adjoint64(v, t, rays, res, w)
    # a ray's 32-bit origin moves its barycentrics by eps * |o| / (size of a triangle),
    # about 6e-8 * 2 / 0.06, and the sums add a few eps (the same formula in 32-bit
    # numpy with 64-bit sums is 5e-7 to 8e-7 off): below 1e-5 of the norm
    err = np.linalg.norm(grad.cpu().numpy().astype(np.float64) - exp) / np.linalg.norm(exp)
    assert err < 1e-5


def _fan(k, corner):
    """k triangles around one vertex, which is their corner `corner`."""
    a = 2 * np.pi * np.arange(k) / k
    v = np.concatenate([[[0.5, 0.5, 0.0]], np.stack([0.5 + 0.7 * np.cos(a), 0.5 + 0.7 * np.sin(a),
                                                      0.05 * np.sin(3 * a)], 1)]).astype(np.float32)
    i = np.arange(k)
    t = np.stack([np.zeros(k, int), 1 + i, 1 + (i + 1) % k], 1)
    return v, np.roll(t, corner, axis=1).astype(np.int32).copy()


@pytest.mark.parametrize("corner", [0, 1, 2])
@pytest.mark.parametrize("k,n", [(3, 8191), (5, 20001), (64, 4099)])
def test_adjoint_around_a_vertex(ctx, k, n, corner):
    """Rays on the triangles of a fan in no order, so that a warp's triangles share a
    vertex: many rays a vertex (both branches of the rule for coarse meshes) and few."""
    v, t = _fan(k, corner)
    rng = np.random.default_rng(k + corner)
    tri = rng.integers(0, k, n)
    uv = rng.uniform(0.1, 0.45, (n, 2))
    p = v[t[tri]].astype(np.float64)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 4:7] = rng.normal(size=(n, 3)) * 0.1 + [0, 0, -1]
    rays[:, :3] = uv[:, :1] * p[:, 0] + uv[:, 1:] * p[:, 1] + (1 - uv.sum(1, keepdims=True)) * p[:, 2] - rays[:, 4:7]
    res = np.zeros((n, 4), np.int32)
    res[:, 0] = np.where(rng.random(n) < 0.05, -1, tri)
    res[:, 1] = np.ones(n, np.float32).view(np.int32)
    res[:, 2:] = uv.astype(np.float32).view(np.int32)
    w = rng.standard_normal((n, 3)).astype(np.float32)
    grad = ctx.adjoint(dev(v), dev(t), dev(rays), dev(res), dev(w))
    ctx.check()
    exp = oracle.adjoint64(v, t, rays, res, w)
    # as in test_adjoint_groups_and_alignment, with triangles of 0.07 and more
    err = np.linalg.norm(grad.cpu().numpy().astype(np.float64) - exp) / np.linalg.norm(exp)
    assert err < 1e-5


def test_adjoint_fan_costs_little_more(ctx):
    """Rays on 4,096 triangles around one vertex take no more than eight times as long as
    on as many of a grid (twice, as measured; 50 times when every lane added to the
    vertex by itself)."""
    m = 1 << 20
    rng = np.random.default_rng(1)
    y, x = np.meshgrid(np.arange(46), np.arange(46), indexing="ij")
    a = (y[:-1, :-1] * 46 + x[:-1, :-1]).reshape(-1)
    grid = (np.stack([x, y, np.sin(x + y)], -1).reshape(-1, 3).astype(np.float32),
            np.stack([a, a + 1, a + 47, a, a + 47, a + 46], -1).reshape(-1, 3).astype(np.int32))
    ms = {}
    for name, (v, t) in (("fan", _fan(4096, 0)), ("grid", grid)):
        res = np.zeros((m, 4), np.int32)
        res[:, 0] = rng.integers(0, len(t), m)
        res[:, 2:] = np.float32(0.25).view(np.int32)
        rays = np.zeros((m, 8), np.float32)
        rays[:, 4:7] = [0.1, 0.2, -1]
        V, T, R, H = dev(v), dev(t), dev(rays), dev(res)
        W, G = torch.ones((m, 3), device="cuda"), torch.zeros_like(V)
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        got = []
        for _ in range(7):
            e[0].record()
            ctx.adjoint(V, T, R, H, W, dl_dverts=G)
            e[1].record()
            e[1].synchronize()
            got.append(e[0].elapsed_time(e[1]))
        ms[name] = sorted(got)[3]
    ctx.check()
    assert ms["fan"] < 8 * ms["grid"], ms
