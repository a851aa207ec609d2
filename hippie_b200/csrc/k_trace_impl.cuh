// The persistent-warp binary-BVH tracer, shared by two translation units that
// differ only in their reciprocal and compiler flags:
//   k_trace.cu      HP_TRACE_RCP(x) = __frcp_rn(x), IEEE round-to-nearest (the
//                   library's default arithmetic, reproduced bit for bit by the
//                   CPU oracle);
//   k_refarith.cu   HP_TRACE_RCP(x) = 1.0f / x compiled with -use_fast_math:
//                   the quotient and denormal flushing of the reference's
//                   fast-math build (gpu/HipCompiler.cpp:127-129), so that its
//                   hits can be reproduced bit for bit. Every other operation
//                   here is an explicit __fmaf_rn / __fmul_rn / __fadd_rn,
//                   which that flag does not contract further.
// Included inside an anonymous namespace after hp_device.cuh / hp_internal.h,
// with HP_TRACE_RCP defined.
#ifndef HP_TRACE_RCP
#error "define HP_TRACE_RCP before including k_trace_impl.cuh"
#endif

constexpr int TRACE_BLOCK = 128;
constexpr int STACK = 64;         // traversal stack entries per ray: SST in shared memory, the rest local
constexpr int SENTINEL = 0x76543210;
constexpr int TRAVERSAL_LIMIT = 1 << 22;  // visits per ray before the ray is abandoned with an error

struct ray_state {
    float ox, oy, oz, tmin, dx, dy, dz;
    float idx_, idy, idz, oodx, oody, oodz;
    float hit_t;
    int hit;       // woop / leaf-ordered reference index of the closest hit, -1 if none
    int nodes, tris;
};

// One 32-byte read-only load (sm_100 vector width); p must be 32-byte aligned.
__device__ __forceinline__ void ld32(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}

__device__ __forceinline__ float safe_rcp(float d) {
    // idir = 1 / (|d| > 2^-80 ? d : copysign(2^-80, d)) (HipTracerBinKernels.cu:83-86)
    const float ooeps = 8.2718061255302767e-25f;  // 2^-80
    return HP_TRACE_RCP(fabsf(d) > ooeps ? d : copysignf(ooeps, d));
}

// Index of the segment containing element g: the last m with off[m] <= g.
__device__ __forceinline__ int seg_search(const int64_t* __restrict__ off, int num_segs, int64_t g) {
    int lo = 0, hi = num_segs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// What bounds the tracer is, first, how many lanes of a warp do the same thing
// (6.3 of 32 per instruction when every lane ran its own loops over nodes and
// over the triangles of its leaves, a warp in any number of pieces) and then the
// L1's request rate: a 64-byte node is two requests of one line a lane, about 2.1
// cycles of an SM's L1 when it comes from L2 and 1.4 when it hits, and a bounce
// ray of the 4.2 M-triangle scene takes 79 nodes, 6 leaves and 14 triangles. So a
// warp stays in one piece and takes three kinds of turns, all 32 lanes together,
// decided by ballots:
//   * nodes: every lane at an interior node does one. The first leaf that a lane
//     meets is postponed and the lane goes on from its stack; at a second one it
//     waits. The turn ends when fewer than LEAST lanes have an interior node and no
//     postponed leaf, so that a hit is found, and shortens the ray, soon;
//   * triangles: every lane with a postponed leaf tests one triangle, until fewer
//     than LEAST lanes have one (or none, once the rays have run out and no lane has a
//     node to go on with);
//   * new rays: once FETCH lanes are without work.
// A stack entry is the child alone. With its entry distance beside it, entries beyond
// the hit found since could be dropped at the pop; that saved no time (bounce rays 19.6
// ms with it, 19.5 without), and for a leaf it is wrong: a leaf's triangles are tested
// whatever its box, whose rounded slabs may lie beyond a nearer or equal hit in it.
//
// LEAST decides more than time. Of two hits nearer to each other than a slab's rounding
// (on the edge that two triangles share) a ray misses the nearer one if the other was
// tested before the nearer one's boxes were, and short node turns test sooner. Against
// a tracer that gives boxes a slack, rays that missed the nearer hit in 360 frames of
// 2.07 M primary rays and in 360 times 4.2 M sphere rays on terrains: every lane in
// loops of its own, as in the reference, 122 and 217; LEAST 1: 122 and 223; 2: 132, 228;
// 3: 126, 232; 4: 128, 235; 16: 151, 280. And it is other rays: of runs over the 4.2 M, 5 %
// differ in a ray between two runs of either order (which rays share a warp is decided as
// they come), 7 % between loops and LEAST 1, 20 % between loops and 4. So where triangles
// share vertices leaves are tested late (LEAST 1), which returns what has always been
// returned, and sooner elsewhere, where such pairs of hits do not come up. A build looks
// whether they do (hp_bvh_info::lone); a batch's warp goes by the meshes whose rays it has.
// A visibility ray has no nearest hit to miss.
//
// Measured on a B200, every lane in loops of its own -> now: 16.8 M bounce rays 28.4 -> 18.2 ms,
// 43 M rays over 256 meshes 42.4 -> 27.3, 4 M sorted rays 3.84 -> 2.87, 1.3 M rays in 10,763 triangles
// 0.73 -> 0.60, 8.4 M rays in 33 M triangles 44.5 -> 45.6 (late, as LARGE_REFS says); late, 2.07 M
// primary rays 0.76 -> 0.65, 4.2 M downward rays 2.28 -> 2.13, 4.2 M bounce rays on a terrain 3.12 ->
// 2.63. Bounce, sorted and batch rays at LEAST 1: 22.9, 3.23 and 32; 4: 18.9, 2.90 and 28.0; 16: 19.5,
// 3.00 and 27.9. FETCH 12 instead of 16: bounce rays 3 % faster, downward ones 6 % slower and a large
// tree's 4 %; 20: the other way round.
// Packed FP32 for the slabs and 32-byte loads of two Woop rows were slower or no faster.
template <bool ANY_HIT>
struct turns {
    static constexpr int LEAST = ANY_HIT ? 12 : 8, FETCH = 16;
};
// CTAs per SM that the kernel is compiled for. Closest hits: 12 (40 registers, some spilled) in
// trees that the L1 does not help much, where bounce rays take 18.2 ms instead of 19.8 at 10 (46
// registers); 10 below SMALL_REFS, where instructions count: 1.3 M rays in 10,763 triangles 0.598
// instead of 0.625 ms, 1 M in 100,003 1.07 instead of 1.12; at 0.5 to 1 M triangles equal.
// Any hit: 1.05 M shadow rays 0.91 ms at 8 and 9, 0.97 at 10, 1.02 at 12. Batch (the
// mesh's bases in the lane, 55 registers): 27.3 ms at 8, 28.9 at 9, 30.0 at 10.
constexpr int CTAS_LARGE = 12, CTAS_SMALL = 10, CTAS_ANY = 9, CTAS_BATCH = 8;
constexpr int64_t SMALL_REFS = 1 << 19;

// BATCH: rays of many meshes in one launch; ray g belongs to the segment whose
// ray range holds it, and the lane traverses that mesh's BVH.
// LATE: leaves are tested late (a batch's warp decides for itself).
template <bool ANY_HIT, bool STATS, bool BATCH, int SST, bool LATE>
__device__ __forceinline__ void trace_rays(
    const float4* __restrict__ rays, int64_t num_rays, int4* __restrict__ results,
    int2* __restrict__ stats, const float4* __restrict__ nodes_all, const float4* __restrict__ woop_all,
    const int32_t* __restrict__ tri_all, int max_nodes_all, int num_refs_all,
    unsigned long long* ray_counter, int* err, const hp_batch_seg* __restrict__ segs,
    const int64_t* __restrict__ ray_off, int num_segs, const int32_t* __restrict__ order, bool late, int* sstack) {
    constexpr int LST = STACK - SST;
    using TURN = turns<ANY_HIT>;
    int lstack[LST];
    const int lane = threadIdx.x & 31;

    ray_state r;
    r.hit_t = 0.0f;
    r.hit = -1;
    int64_t ray = -1;
    int node = SENTINEL;
    int leaf = 0;            // postponed leaf (~index) whose range is not loaded yet, 0 when none
    int tri = 0, tri_end = 0;  // triangles of the postponed leaf still to test
    int sp = 0;
    int steps = 0;           // node + leaf visits of the current ray (bounded)
    bool exhausted = false;  // warp-uniform: the counter has run past the rays
    bool lone = true;        // of the lane's mesh (BATCH)
    int least = LATE ? 1 : TURN::LEAST;  // warp-uniform
    const float4* nodes = nodes_all;
    const float4* woop = woop_all;
    const int32_t* tri_idx = tri_all;
    int max_nodes = max_nodes_all, num_refs = num_refs_all;

    auto pop = [&]() {
        if (sp == 0) {
            node = SENTINEL;
        } else {
            --sp;
            node = sp < SST ? sstack[sp * TRACE_BLOCK] : lstack[sp - SST];
        }
    };

    while (true) {
        // Finished lanes write their results and take new rays (one atomic per warp).
        const bool idle = node == SENTINEL && leaf >= 0 && tri >= tri_end;
        const unsigned idle_mask = __ballot_sync(HP_FULL_MASK, idle);
        if (idle_mask == HP_FULL_MASK || (!exhausted && __popc(idle_mask) >= TURN::FETCH)) {
            if (idle && ray >= 0) {
                if (r.hit < 0) {
                    reinterpret_cast<int2*>(results)[2 * ray] = make_int2(-1, __float_as_int(r.hit_t));
                    if (STATS) stats[ray] = make_int2(0, 0);
                } else {
                    // u and v of the closest hit once more, by the steps of its test
                    const float4 v1 = __ldg(woop + 3 * (int64_t)r.hit + 1), v2 = __ldg(woop + 3 * (int64_t)r.hit + 2);
                    const float hu = __fmaf_rn(
                        r.hit_t, __fmaf_rn(r.dz, v1.z, __fmaf_rn(r.dy, v1.y, __fmul_rn(r.dx, v1.x))),
                        __fmaf_rn(r.oz, v1.z, __fmaf_rn(r.oy, v1.y, __fmaf_rn(r.ox, v1.x, v1.w))));
                    const float hv = __fmaf_rn(
                        r.hit_t, __fmaf_rn(r.dz, v2.z, __fmaf_rn(r.dx, v2.x, __fmul_rn(r.dy, v2.y))),
                        __fmaf_rn(r.oz, v2.z, __fmaf_rn(r.oy, v2.y, __fmaf_rn(r.ox, v2.x, v2.w))));
                    results[ray] = make_int4(__ldg(tri_idx + r.hit), __float_as_int(r.hit_t),
                                             __float_as_int(hu), __float_as_int(hv));
                    if (STATS) stats[ray] = make_int2(r.nodes, r.tris);
                }
                ray = -1;
            }
            if (exhausted) break;  // every lane is idle
            unsigned long long base = 0;
            const int leader = __ffs(idle_mask) - 1;
            if (lane == leader) base = atomicAdd(ray_counter, (unsigned long long)__popc(idle_mask));
            base = __shfl_sync(HP_FULL_MASK, base, leader);
            exhausted = (int64_t)base + __popc(idle_mask) >= num_rays;
            const int64_t slot = (int64_t)base + __popc(idle_mask & ((1u << lane) - 1u));
            if (idle && slot < num_rays) {
                // traceSort: slot k traces ray order[k] (rays in Morton order)
                const int64_t id = order ? (int64_t)__ldg(order + slot) : slot;
                if ((uint64_t)id >= (uint64_t)num_rays) {
                    hp_report(err, HP_DEV_BAD_INDEX, (int)slot);
                } else {
                    ray = id;
                    const float4 o = __ldg(rays + 2 * id), d = __ldg(rays + 2 * id + 1);
                    r.ox = o.x; r.oy = o.y; r.oz = o.z; r.tmin = o.w;
                    r.dx = d.x; r.dy = d.y; r.dz = d.z; r.hit_t = d.w;
                    r.idx_ = safe_rcp(d.x); r.idy = safe_rcp(d.y); r.idz = safe_rcp(d.z);
                    r.oodx = __fmul_rn(o.x, r.idx_);
                    r.oody = __fmul_rn(o.y, r.idy);
                    r.oodz = __fmul_rn(o.z, r.idz);
                    r.hit = -1;
                    r.nodes = r.tris = 0;
                    sp = 0;
                    steps = 0;
                    node = 0;
                    if (BATCH) {
                        const hp_batch_seg& g = segs[seg_search(ray_off, num_segs, id)];
                        lone = g.lone != 0;
                        nodes = nodes_all + 4 * g.node_off;
                        woop = woop_all + 3 * (int64_t)g.tri_off;
                        tri_idx = tri_all + g.tri_off;
                        num_refs = g.n;
                        max_nodes = max(2 * g.n - 1, 3);
                        if (g.n == 0) node = SENTINEL;  // empty mesh: the ray misses
                    }
                }
            }
            if (BATCH)
                least = late || (!ANY_HIT && __any_sync(HP_FULL_MASK, ray >= 0 && !lone)) ? 1 : TURN::LEAST;
        }

        // Interior nodes: one per lane and round.
        bool go = (unsigned)node < (unsigned)SENTINEL;
        unsigned mask = __ballot_sync(HP_FULL_MASK, go);
        while (mask) {
            if (go) {
                if (node >= max_nodes || ++steps > TRAVERSAL_LIMIT) {
                    hp_report(err, HP_DEV_BAD_INDEX, node);
                    node = SENTINEL;
                    leaf = 0;
                    tri = tri_end = 0;
                } else {
                    if (STATS) ++r.nodes;
                    const float4* np = nodes + 4 * (int64_t)node;
                    float4 n0, n1, nz, nm;
                    ld32(np, n0, n1);
                    ld32(np + 2, nz, nm);
                    const float c0lox = __fmaf_rn(n0.x, r.idx_, -r.oodx);
                    const float c0hix = __fmaf_rn(n0.y, r.idx_, -r.oodx);
                    const float c0loy = __fmaf_rn(n0.z, r.idy, -r.oody);
                    const float c0hiy = __fmaf_rn(n0.w, r.idy, -r.oody);
                    const float c0loz = __fmaf_rn(nz.x, r.idz, -r.oodz);
                    const float c0hiz = __fmaf_rn(nz.y, r.idz, -r.oodz);
                    const float c1loz = __fmaf_rn(nz.z, r.idz, -r.oodz);
                    const float c1hiz = __fmaf_rn(nz.w, r.idz, -r.oodz);
                    const float c1lox = __fmaf_rn(n1.x, r.idx_, -r.oodx);
                    const float c1hix = __fmaf_rn(n1.y, r.idx_, -r.oodx);
                    const float c1loy = __fmaf_rn(n1.z, r.idy, -r.oody);
                    const float c1hiy = __fmaf_rn(n1.w, r.idy, -r.oody);
                    const float c0min = fmaxf(fmaxf(fminf(c0lox, c0hix), fminf(c0loy, c0hiy)),
                                              fmaxf(fminf(c0loz, c0hiz), r.tmin));
                    const float c0max = fminf(fminf(fmaxf(c0lox, c0hix), fmaxf(c0loy, c0hiy)),
                                              fminf(fmaxf(c0loz, c0hiz), r.hit_t));
                    const float c1min = fmaxf(fmaxf(fminf(c1lox, c1hix), fminf(c1loy, c1hiy)),
                                              fmaxf(fminf(c1loz, c1hiz), r.tmin));
                    const float c1max = fminf(fminf(fmaxf(c1lox, c1hix), fmaxf(c1loy, c1hiy)),
                                              fminf(fmaxf(c1loz, c1hiz), r.hit_t));
                    const bool t0 = c0max >= c0min, t1 = c1max >= c1min;
                    const int c0 = __float_as_int(nm.x), c1 = __float_as_int(nm.y);
                    const bool swap = t1 && (!t0 || c1min < c0min);
                    node = swap ? c1 : c0;
                    if (t0 && t1) {
                        const int far = swap ? c0 : c1;
                        if (sp < SST) sstack[sp * TRACE_BLOCK] = far;
                        else if (sp < STACK) lstack[sp - SST] = far;
                        else { hp_report(err, HP_DEV_STACK_OVERFLOW, (int)ray); --sp; }
                        ++sp;
                    }
                    if (!t0 && !t1) pop();
                    if (node < 0 && leaf >= 0 && tri >= tri_end) {  // the first leaf is postponed
                        leaf = node;
                        pop();
                    }
                }
            }
            go = (unsigned)node < (unsigned)SENTINEL;
            mask = __ballot_sync(HP_FULL_MASK, go && leaf >= 0 && tri >= tri_end);
            if (__popc(mask) < least) break;
        }

        // Leaves: one triangle per lane and round.
        bool pend = node < 0 || leaf < 0 || tri < tri_end;
        mask = __ballot_sync(HP_FULL_MASK, pend);
        while (mask) {
            if (pend) {
                if (leaf >= 0 && tri >= tri_end) {  // the leaf that the lane stopped at
                    leaf = node;
                    pop();
                }
                if (leaf < 0) {
                    const int li = ~leaf;
                    leaf = 0;
                    tri = tri_end = 0;
                    if (li >= max_nodes || ++steps > TRAVERSAL_LIMIT) {
                        hp_report(err, HP_DEV_BAD_INDEX, li);
                        node = SENTINEL;
                        sp = 0;
                    } else {
                        const int2 lm = __ldg(reinterpret_cast<const int2*>(nodes + 4 * (int64_t)li + 3));
                        if (lm.x < 0 || lm.y > num_refs || lm.x > lm.y) {
                            hp_report(err, HP_DEV_BAD_INDEX, lm.x);
                        } else {
                            tri = lm.x;
                            tri_end = lm.y;
                        }
                    }
                }
                if (tri < tri_end) {
                    if (STATS) ++r.tris;
                    const float4* wp = woop + 3 * (int64_t)tri;
                    const float4 v0 = __ldg(wp);
                    const float4 v1 = __ldg(wp + 1);
                    const float oz = __fmaf_rn(-r.oz, v0.z, __fmaf_rn(-r.oy, v0.y, __fmaf_rn(-r.ox, v0.x, v0.w)));
                    // The roundings of the reference's fast-math tracer, measured
                    // against its output on sm_100a: the chains o.w +- ... are
                    // contracted term by term from the left; of the three-term dot
                    // products d.w, the denominator and the v term fuse the x
                    // product over the rounded y product, the u term the y product
                    // over the rounded x product (nvcc's choice depends on context).
                    const float den = __fmaf_rn(r.dz, v0.z, __fmaf_rn(r.dx, v0.x, __fmul_rn(r.dy, v0.y)));
                    const float t = __fmul_rn(oz, HP_TRACE_RCP(den));
                    bool closer = t < r.hit_t;
                    if (!closer && t == r.hit_t && r.hit >= 0)
                        closer = __ldg(tri_idx + tri) < __ldg(tri_idx + r.hit);
                    if (t > r.tmin && closer) {
                        const float ox = __fmaf_rn(r.oz, v1.z, __fmaf_rn(r.oy, v1.y, __fmaf_rn(r.ox, v1.x, v1.w)));
                        const float dx = __fmaf_rn(r.dz, v1.z, __fmaf_rn(r.dy, v1.y, __fmul_rn(r.dx, v1.x)));
                        const float u = __fmaf_rn(t, dx, ox);
                        if (u >= 0.0f) {
                            const float4 v2 = __ldg(wp + 2);
                            const float oy = __fmaf_rn(r.oz, v2.z, __fmaf_rn(r.oy, v2.y, __fmaf_rn(r.ox, v2.x, v2.w)));
                            const float dy = __fmaf_rn(r.dz, v2.z, __fmaf_rn(r.dx, v2.x, __fmul_rn(r.dy, v2.y)));
                            const float v = __fmaf_rn(t, dy, oy);
                            if (v >= 0.0f && __fadd_rn(u, v) <= 1.0f) {
                                r.hit_t = t;
                                r.hit = tri;
                                if (ANY_HIT) { node = SENTINEL; sp = 0; tri = tri_end; }
                            }
                        }
                    }
                    ++tri;
                }
            }
            pend = node < 0 || leaf < 0 || tri < tri_end;
            mask = __ballot_sync(HP_FULL_MASK, pend);
            if (__popc(mask) < least &&
                !(exhausted && mask && !__any_sync(HP_FULL_MASK, (unsigned)node < (unsigned)SENTINEL)))
                break;
        }
    }
}

template <bool ANY_HIT, bool STATS, bool BATCH, int SST, int CTAS>
__global__ void __launch_bounds__(TRACE_BLOCK, CTAS) k_trace(
    const float4* __restrict__ rays, int64_t num_rays, int4* __restrict__ results,
    int2* __restrict__ stats, const float4* __restrict__ nodes_all, const float4* __restrict__ woop_all,
    const int32_t* __restrict__ tri_all, int max_nodes_all, int num_refs_all,
    unsigned long long* ray_counter, int* err, const hp_batch_seg* __restrict__ segs,
    const int64_t* __restrict__ ray_off, int num_segs, const int32_t* __restrict__ order,
    const hp_bvh_info* __restrict__ info, bool late) {
    __shared__ int s_stack[SST * TRACE_BLOCK];
    int* sstack = s_stack + threadIdx.x;
    // One body a kind of mesh: with one body and its limit in a register bounce rays take
    // 20.0 ms, not 19.1.
    if (!BATCH && (late || (!ANY_HIT && __ldg(&info->lone) == 0)))
        trace_rays<ANY_HIT, STATS, BATCH, SST, true>(rays, num_rays, results, stats, nodes_all, woop_all, tri_all,
                                                     max_nodes_all, num_refs_all, ray_counter, err, segs, ray_off,
                                                     num_segs, order, late, sstack);
    else
        trace_rays<ANY_HIT, STATS, BATCH, SST, false>(rays, num_rays, results, stats, nodes_all, woop_all, tri_all,
                                                      max_nodes_all, num_refs_all, ray_counter, err, segs, ray_off,
                                                      num_segs, order, late, sstack);
}

// Persistent CTAs: the tuned number per SM, or as many as fit.
int64_t trace_resident(const hp_ctx* ctx, int per_sm) {
    int k = std::max(per_sm, 1);
    if (ctx->tune.trace_ctas_per_sm > 0) k = std::min(k, (int)ctx->tune.trace_ctas_per_sm);
    return (int64_t)ctx->sm_count * k;
}
int trace_grid(const hp_ctx* ctx, int per_sm, int64_t num_rays) {
    const int64_t grid = std::min<int64_t>(trace_resident(ctx, per_sm), (num_rays + TRACE_BLOCK - 1) / TRACE_BLOCK);
    return (int)std::max<int64_t>(grid, 1);
}

// A launch that has no two rays for a lane lasts as long as its slowest warps: their lanes
// take every turn they can (LEAST 1) instead of waiting for a fuller one, on any mesh (131,072
// rays in 1.7 M triangles on a B200 587 -> 568 us, 1,000 visibility rays on a terrain 89 -> 72;
// as a rule for 4 or 8 rays a lane 1 M visibility rays lose 6 %).
bool few_rays(const hp_ctx* ctx, int per_sm, int64_t num_rays) {
    return num_rays < 2 * trace_resident(ctx, per_sm) * TRACE_BLOCK;
}

// Closest hits of rays in an order of their own in trees far beyond the L2 wait for DRAM, and
// wait less with leaves tested late, while more lanes have a node to ask for: 8.4 M sphere
// rays, late and not, in 8 M triangles 14.5 and 14.0 ms, 16 M 25.2 and 25.9, 33 M 45.6 and 47.6
// (25.3 and 44.5 with every lane in loops of its own); in ray Morton order 14.5 and 12.5 for
// 16 M, 23.9 and 21.5 for 33 M.
constexpr int64_t LARGE_REFS = 12 << 20;

template <bool A, bool S, int SST, int CTAS>
hp_status launch_t(hp_ctx* ctx, const hp_bvh_impl* b, int64_t n_refs, const float* rays,
                   int64_t num_rays, int32_t* results, int32_t* stats, unsigned long long* counter,
                   const int32_t* order, cudaStream_t s) {
    int per_sm = 0;
    HP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace<A, S, false, SST, CTAS>, TRACE_BLOCK, 0));
    const int max_nodes = (int)std::max<int64_t>(2 * b->capacity - 1, 3);
    k_trace<A, S, false, SST, CTAS><<<trace_grid(ctx, per_sm, num_rays), TRACE_BLOCK, 0, s>>>(
        reinterpret_cast<const float4*>(rays), num_rays, reinterpret_cast<int4*>(results),
        reinterpret_cast<int2*>(stats), reinterpret_cast<const float4*>(b->nodes), b->woop, b->tri_idx,
        max_nodes, (int)n_refs, counter, ctx->d_status, nullptr, nullptr, 0, order, b->info,
        few_rays(ctx, per_sm, num_rays) || (!A && !order && n_refs >= LARGE_REFS));
    HP_CUDA(cudaGetLastError());
    hp_count_launch();
    hp_mark(ctx, s, "trace");
    return HP_OK;
}

template <bool A, bool S, int SST>
hp_status launch_size(hp_ctx* ctx, const hp_bvh_impl* b, int64_t n_refs, const float* rays,
                      int64_t num_rays, int32_t* results, int32_t* stats, unsigned long long* counter,
                      const int32_t* order, cudaStream_t s) {
    if constexpr (A)
        return launch_t<A, S, SST, CTAS_ANY>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
    else if (n_refs < SMALL_REFS)
        return launch_t<A, S, SST, CTAS_SMALL>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
    else
        return launch_t<A, S, SST, CTAS_LARGE>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
}

template <bool A, bool S>
hp_status launch_st(hp_ctx* ctx, const hp_bvh_impl* b, int64_t n_refs, const float* rays,
                    int64_t num_rays, int32_t* results, int32_t* stats, unsigned long long* counter,
                    const int32_t* order, cudaStream_t s) {
    switch (ctx->tune.trace_stack) {
        case 8: return launch_size<A, S, 8>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
        case 32: return launch_size<A, S, 32>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
        default: return launch_size<A, S, 16>(ctx, b, n_refs, rays, num_rays, results, stats, counter, order, s);
    }
}
