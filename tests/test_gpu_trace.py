"""GPU closest-hit traversal against the CPU oracle: results bit-identical
(triangle id, t, u, v), stats identical, any-hit semantics (sm_100a)."""
import numpy as np
import pytest
import torch

import hippie_b200 as hp
import oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _setup(ctx, kind, n, n_rays, bits, seed=0):
    if kind == "uniform":
        v, t = hp.gen.uniform_mesh(seed + 1, n)
        rays = hp.gen.rays_targeted(seed + 2, n_rays)
    else:
        v, t = hp.gen.clustered_mesh(seed + 1, n, clusters=1024)
        lo, hi = v.min(0), v.max(0)
        rays = hp.gen.rays_sphere(seed + 2, n_rays, np.concatenate([lo, hi]))
    bvh = ctx.build(dev(v), dev(t), hp.BuildParams(morton_bits=bits))
    bvh.sync()
    return v, t, rays, bvh


@pytest.mark.parametrize("kind,n,n_rays,bits", [("uniform", 65536, 1 << 20, 30),
                                                ("clustered", 262144, 1 << 20, 60)])
def test_trace_bit_exact(ctx, kind, n, n_rays, bits):
    v, t, rays, bvh = _setup(ctx, kind, n, n_rays, bits)
    R = dev(rays)
    res = torch.zeros((n_rays, 4), dtype=torch.int32, device="cuda")
    st = torch.zeros((n_rays, 2), dtype=torch.int32, device="cuda")
    ctx.trace(bvh, R, results=res, stats=st)
    ctx.check()
    nodes, woop, tri = bvh.download()
    exp, est = oracle.trace(nodes, woop, tri, rays, stats=True)
    got = res.cpu().numpy()
    np.testing.assert_array_equal(got, exp)
    # Counters: postponed leaves make the GPU's visit order depend on the warp,
    # so node / triangle counts are compared in aggregate, not per ray.
    gst = st.cpu().numpy()
    hit = exp[:, 0] >= 0
    assert np.all(gst[~hit] == 0) and np.all(gst[hit] > 0)
    for k in range(2):
        assert abs(gst[hit, k].mean() / est[hit, k].mean() - 1.0) < 0.15
    hits = (got[:, 0] >= 0).mean()
    assert 0.05 < hits < 1.0
    # plain trace (no stats) gives the same results
    res2 = torch.zeros_like(res)
    ctx.trace(bvh, R, results=res2)
    assert torch.equal(res, res2)


def test_trace_vs_double_brute_force(ctx):
    v, t, rays, bvh = _setup(ctx, "uniform", 4000, 20000, 60, seed=5)
    got = ctx.trace(bvh, dev(rays)).cpu().numpy()
    bf = oracle.brute64(v, t, rays)
    hit = got[:, 0] >= 0
    both = hit & (bf[:, 0] >= 0)
    assert np.mean(hit == (bf[:, 0] >= 0)) > 0.999
    assert np.mean(got[both, 0] == bf[both, 0]) > 0.999
    tuv = got[both, 1:].view(np.float32).astype(np.float64)
    err = np.abs(tuv - bf[both, 1:]) / np.maximum(1.0, np.abs(bf[both, 1:]))
    # t is accurate to a few ulps; the FP32 Woop test computes u and v as a
    # difference of terms ~1/triangle size, so against exact barycentrics they
    # carry ~1e-5 absolute error (as the reference's own Woop test does).
    assert np.median(err[:, 0]) < 1e-6 and np.quantile(err[:, 0], 0.999) < 1e-4
    assert np.quantile(err[:, 1:], 0.99) < 1e-3


def test_any_hit_and_limits(ctx):
    v, t, rays, bvh = _setup(ctx, "uniform", 50000, 100000, 30, seed=9)
    R = dev(rays)
    closest = ctx.trace(bvh, R).cpu().numpy()
    anyh = torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda")
    ctx.trace(bvh, R, results=anyh, any_hit=True)
    anyh = anyh.cpu().numpy()
    np.testing.assert_array_equal(anyh[:, 0] >= 0, closest[:, 0] >= 0)
    # any hit: some intersected triangle, never closer than the closest one
    h = anyh[:, 0] >= 0
    assert np.all(anyh[h, 1].view(np.float32) >= closest[h, 1].view(np.float32))
    bf = oracle.brute64(v, t, rays[h][:2000])
    for i, row in enumerate(anyh[h][:2000]):
        p = v[t[row[0]]].astype(np.float64)
        ok, tuv = oracle.intersect64(p[0], p[1], p[2], rays[h][i, :3], rays[h][i, 4:7])
        assert ok and abs(tuv[0] - row[1:2].view(np.float32)[0]) <= 1e-4 * max(1.0, tuv[0]), i
    assert np.all(bf[:, 0] >= 0)
    nodes, woop, tri = bvh.download()
    # tmin / tmax windows
    r2 = rays.copy()
    r2[:, 3] = 0.3
    r2[:, 7] = 1.2
    got = ctx.trace(bvh, dev(r2), results=torch.zeros((r2.shape[0], 4), dtype=torch.int32, device="cuda"))
    exp = oracle.trace(nodes, woop, tri, r2)
    np.testing.assert_array_equal(got.cpu().numpy(), exp)
    tt = exp[exp[:, 0] >= 0, 1].view(np.float32)
    assert np.all((tt > 0.3) & (tt < 1.2))
    miss = exp[:, 0] < 0
    assert np.all(exp[miss, 1].view(np.float32) == np.float32(1.2))


def test_axis_aligned_rays(ctx):
    """Direction components of exactly zero take the 2^-80 reciprocal path."""
    v, t = hp.gen.uniform_mesh(3, 20000)
    bvh = ctx.build(dev(v), dev(t), hp.BuildParams(morton_bits=30))
    rng = np.random.default_rng(0)
    n = 30000
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(0, 1, (n, 3))
    axis = rng.integers(0, 3, n)
    sign = rng.choice([-1.0, 1.0], n)
    rays[np.arange(n), 4 + axis] = sign
    rays[np.arange(n), axis] = np.where(sign > 0, -0.5, 1.5)
    rays[:, 7] = np.inf
    got = ctx.trace(bvh, dev(rays)).cpu().numpy()
    nodes, woop, tri = bvh.download()
    exp = oracle.trace(nodes, woop, tri, rays)
    np.testing.assert_array_equal(got[:, :2], exp[:, :2])
    h = exp[:, 0] >= 0
    np.testing.assert_array_equal(got[h], exp[h])


@pytest.mark.parametrize("slope", [1.0, 1e-3, 1e-5])
@pytest.mark.parametrize("arith,layout", [("ieee", 2), ("reference", 2), ("ieee", 4), ("ieee", 8)])
def test_leaves_of_one_plane(arith, layout, slope):
    """Overlapping triangles of one axis-aligned plane, in leaves whose boxes are all
    looked at before any hit is known (children of the root; in the binary tree also of
    the root's first child, which a ray visits first). A leaf's triangles are tested
    whatever its flat box's rounded slabs say of a hit found since, so a ray returns
    the nearest of them, of equal ones the lowest id, with and without statistics: what
    the triangles return one by one. `slope` scales the rays' components along the
    plane, down to rays nearly along the axis."""
    c = hp.Context(0)
    c.set_arithmetic(arith)
    rng = np.random.default_rng(layout)
    n, m = max(layout, 3), 1 << 14
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) + np.array([0, 2.1, 4.2]) + rng.uniform(-0.3, 0.3, (n, 3))
    rad = rng.uniform(0.3, 0.9, (n, 3))
    rad[:] = rad.mean(1, keepdims=True)
    at = np.full((n, 1), 0.45)
    at[-1] = 0.65  # the last Morton code
    v = np.stack([at + rad * np.cos(ang), at + rad * np.sin(ang), np.full_like(rad, 0.3)], -1)
    v = v.reshape(-1, 3).astype(np.float32)
    t = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    rays = np.zeros((m, 8), np.float32)
    rays[:, :2] = rng.uniform(0.3, 0.7, (m, 2))
    rays[:, 2] = rng.uniform(0.5, 1.5, m)
    rays[:, 4:6] = slope * rng.uniform(-0.3, 0.3, (m, 2))
    rays[:, 6] = 0.3 - rays[:, 2]
    rays[:, 7] = 10
    R = dev(rays)
    p = hp.BuildParams(method="lbvh", morton_bits=60, layout=layout, adaptive_leaf=0, max_leaf_size=1)

    def hits(ctx, bvh, **kw):
        out = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
        ctx.trace(bvh, R, results=out, **kw)
        ctx.check()
        return out.cpu().numpy()

    bvh = c.build(dev(v), dev(t), p)
    bvh.sync()
    assert bvh.c.num_interior == (2 if layout == 2 else 1)
    if layout == 2:
        assert bvh.download()[0][0, 12] == 1 and bvh.download()[0][0, 13] < 0
    got = hits(c, bvh)
    want = np.zeros((m, 4), np.int32)
    want[:, 0], want[:, 1] = -1, rays[:, 7].view(np.int32)
    for i in range(n):  # in the order of the ids: a later one has to be nearer
        one = hits(c, c.build(dev(v[3 * i:3 * i + 3]), dev(t[:1]), p))
        nearer = (one[:, 0] >= 0) & (one[:, 1].view(np.float32) < want[:, 1].view(np.float32))
        want[nearer] = one[nearer]
        want[nearer, 0] = i
    assert (want[:, 0] >= 0).mean() > 0.5 and len(np.unique(want[:, 0])) > 1
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(hits(c, bvh, stats=torch.zeros((m, 2), dtype=torch.int32, device="cuda")), want)
    c.close()


@pytest.mark.parametrize("layout", [2, 4, 8])
def test_one_order_for_every_copy_of_a_mesh(ctx, layout):
    """A terrain with shared vertices, with vertices of its own per triangle, and with
    unreferenced vertices behind it, and its BVH in reserved storage: the tracer walks
    all four alike. How many nodes rays visit tells the order of their turns (how often a
    hit shortens the ray before the next node), and the hits are the same."""
    v, t = hp.gen.heightfield(3, 200, 300)
    n, m = len(t), 1 << 20
    own = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    meshes = {"shared": (v, t), "own": (v[t].reshape(-1, 3), own), "padded": (np.concatenate([v] * 6), t)}
    R = dev(hp.gen.rays_sphere(4, m, np.concatenate([v.min(0), v.max(0)])))
    p = hp.BuildParams(method="lbvh", morton_bits=60, layout=layout)
    bvhs = {k: ctx.build(dev(a), dev(b), p) for k, (a, b) in meshes.items()}
    for b in bvhs.values():
        b.sync()
    src = bvhs["own"]
    bvhs["reserved"] = hp.BVH.reserve(ctx, n, layout)
    for to, frm in zip(bvhs["reserved"].arrays(), src.arrays()):
        to.copy_(frm)
    bvhs["reserved"].set_info(src.c.num_interior, src.c.num_leaf, src.c.scene_box, src.c.morton_scale)
    visits, hits = {}, {}
    for k, b in bvhs.items():
        res = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
        st = torch.zeros((m, 2), dtype=torch.int32, device="cuda")
        ctx.trace(b, R, results=res, stats=st)
        ctx.check()
        visits[k], hits[k] = float(st[:, 0].double().sum()), res
    for k in bvhs:
        # runs of one order differ by the rays that happen to share a warp: by less than 1e-4
        assert abs(visits[k] / visits["shared"] - 1) < 2e-3, visits
        # two hits on a shared edge, within a slab's rounding: a few in 1e8 rays
        assert int((hits[k][:, 0] != hits["shared"][:, 0]).sum()) <= 3, k


@pytest.mark.parametrize("n,pair", [(3000, 2998), (8191, 17), (8192, 4096), (30000, 4)])
def test_a_shared_vertex_is_found(ctx, n, pair):
    """Triangles with vertices of their own are traced with short turns, those of a mesh in
    which a triangle looked at (every one up to 8,191, of 30,000 every fourth) has a vertex
    in common with the next late, as trees are that no build has looked over. The nodes
    that rays visit tell which; the hits are the same."""
    m = 1 << 19
    v, t = hp.gen.uniform_mesh(n, n, 0.02)
    w = v.copy()
    w[3 * (pair + 1)] = w[3 * pair + 2]
    R = dev(hp.gen.rays_sphere(4, m, np.concatenate([v.min(0), v.max(0)])))
    p = hp.BuildParams(method="lbvh", morton_bits=60)

    def visits(bvh):
        res = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
        st = torch.zeros((m, 2), dtype=torch.int32, device="cuda")
        ctx.trace(bvh, R, results=res, stats=st)
        ctx.check()
        return float(st[:, 0].double().sum()), res

    for verts, late in ((v, False), (w, True)):
        built = ctx.build(dev(verts), dev(t), p)
        built.sync()
        known = hp.BVH.reserve(ctx, n)
        for to, frm in zip(known.arrays(), built.arrays()):
            to.copy_(frm)
        known.set_info(built.c.num_interior, built.c.num_leaf, built.c.scene_box, built.c.morton_scale)
        (a, hits_a), (b, hits_b) = visits(built), visits(known)
        assert torch.equal(hits_a, hits_b)
        print(n, late, a / b)
        assert (abs(a / b - 1) < 1e-3) if late else (a / b < 1 - 3e-3), (a, b)


def test_batch_of_both_kinds(ctx):
    """A batch whose warps trace meshes with and without shared vertices gives every mesh's
    own hits."""
    meshes = [hp.gen.uniform_mesh(5, 2000), hp.gen.heightfield(6, 40, 30), hp.gen.uniform_mesh(7, 300),
              hp.gen.heightfield(8, 9, 7)]
    counts = [5000, 77, 4001, 3000]
    p = hp.BuildParams(method="lbvh", morton_bits=30)
    batch = hp.Batch(ctx, [(dev(v), dev(t)) for v, t in meshes], counts, p)
    rays = [hp.gen.rays_sphere(11 + i, k, np.concatenate([v.min(0), v.max(0)]))
            for i, ((v, t), k) in enumerate(zip(meshes, counts))]
    res = torch.zeros((sum(counts), 4), dtype=torch.int32, device="cuda")
    batch.build(graph=False)
    batch.trace(dev(np.concatenate(rays)), results=res, graph=False)
    ctx.check()
    at = 0
    for (v, t), r in zip(meshes, rays):
        one = torch.zeros((len(r), 4), dtype=torch.int32, device="cuda")
        ctx.trace(ctx.build(dev(v), dev(t), p), dev(r), results=one)
        assert torch.equal(res[at:at + len(r)], one)
        at += len(r)
    batch.close()


@pytest.mark.parametrize("ctas", [0, 5])
@pytest.mark.parametrize("layout", [2, 4, 8])
def test_launches_of_few_and_many_rays_agree(ctx, layout, ctas):
    """Just below and at two rays a lane of the CTAs that are launched (10 or 8 per SM, or what
    trace_ctas_per_sm says), and in chunks far below it: the same hits, of a mesh whose
    triangles share vertices and of one whose do not."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = 2 * sms * 128 * (ctas or (10 if layout == 2 else 8))
    ctx.set_tune(trace_ctas_per_sm=ctas)
    try:
        for v, t in (hp.gen.heightfield(3, 120, 150), hp.gen.uniform_mesh(4, 30000)):
            rays = hp.gen.rays_sphere(5, m, np.concatenate([v.min(0), v.max(0)]))
            bvh = ctx.build(dev(v), dev(t), hp.BuildParams(method="lbvh", morton_bits=60, layout=layout))
            R, got = dev(rays), []
            for cuts in ([0, m], [0, m - 1, m], list(range(0, m, 50021)) + [m]):
                res = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
                for a, b in zip(cuts, cuts[1:]):
                    ctx.trace(bvh, R[a:b], results=res[a:b])
                got.append(res)
            ctx.check()
            for other in got[1:]:
                # on a shared edge, within a slab's rounding: a few in 1e8 rays
                assert int((other[:, 0] != got[0][:, 0]).sum()) <= 2
    finally:
        ctx.reset_tune()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19])
def test_both_sizes_of_tracer(ctx, n):
    """Around the tree size where closest hits go to the tracer of more CTAs per SM."""
    v, t, rays, bvh = _setup(ctx, "uniform", n, 50000, 60, seed=3)
    got = ctx.trace(bvh, dev(rays), results=torch.zeros((len(rays), 4), dtype=torch.int32, device="cuda"))
    ctx.check()
    np.testing.assert_array_equal(got.cpu().numpy(), oracle.trace(*bvh.download(), rays))
