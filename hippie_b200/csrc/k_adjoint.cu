// Closest-hit adjoint and refit-only BVH update.
//
// Adjoint: a hit satisfies O + t D = u v0 + v v1 + (1-u-v) v2 (u weights v0 and
// v weights v1, the barycentric convention of rt/HipUtil.h:190-195), i.e.
// A x = O - v2 with A = [v0-v2, v1-v2, -D] and x = (u, v, t). Differentiating,
// dx/dv0 = -u A^-1, dx/dv1 = -v A^-1, dx/dv2 = -(1-u-v) A^-1, so with
// q = A^-T (dL/du, dL/dv, dL/dt):
//   dL/dv0 = -u q,  dL/dv1 = -v q,  dL/dv2 = -(1-u-v) q,
// and A^-T g = (g_u (b x c) + g_v (c x a) + g_t (a x b)) / det(A) for A = [a b c].
// Lanes of a warp whose rays hit the same triangle add their contributions with
// shuffles first, and triangles around a vertex theirs for it, so each costs one set of
// reductions per warp, two requests a vertex. Bound by the reductions' and gathers'
// requests. The sums run over all groups at once with full-warp shuffles: summing a group at
// a time under its own mask ran a warp's groups one after another (4.2 M rays on a
// 1 M-triangle heightfield 0.366 -> 0.092 ms).
//
// Refit: HipBVH::update (rt/bvh/HipBVH.cpp:472-477) = woopifyTriangles +
// refitLeavesBin + refitInteriorsBin (rt/bvh/HipBVHKernels.cu:240-326). The
// reference launches refitLeaves with 4 of its 6 arguments (HipBVH.cpp:43-48);
// this version passes the mesh, so leaf boxes come from the current vertices.
#include <cuda_runtime.h>
#include "hp_device.cuh"
#include "hp_internal.h"

namespace {

constexpr int AB = 256;

__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
    return make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                       __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float dot3(float3 a, float3 b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}
// g0 * x + g1 * y + g2 * z
__device__ __forceinline__ float comb3(float g0, float x, float g1, float y, float g2, float z) {
    return __fmaf_rn(g2, z, __fmaf_rn(g1, y, __fmul_rn(g0, x)));
}

// dverts[3 idx .. 3 idx + 2] += (x, y, z): the 8-byte aligned two of the three
// in one reduction, the other in a second one.
__device__ __forceinline__ void add3(float* __restrict__ dverts, int idx, float x, float y, float z) {
    float* p = dverts + 3 * (int64_t)idx;
    const bool hi = (reinterpret_cast<uintptr_t>(p) & 4u) != 0;
    asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(hi ? p + 1 : p), "f"(hi ? y : x),
                 "f"(hi ? z : y)
                 : "memory");
    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(hi ? p : p + 2), "f"(hi ? x : z) : "memory");
}

// Sums x over the lanes with the same id (no lane with a negative one); the lowest of them
// gets the sum and true. As many rounds as the largest group has halvings: every round,
// each remaining lane of a group takes its next one's sums, and every second lane drops
// out. All 32 lanes take part in every shuffle, whatever their groups.
template <int C>
__device__ __forceinline__ bool join(int id, float (&x)[C]) {
    const int lane = threadIdx.x & 31;
    const unsigned grp = __match_any_sync(HP_FULL_MASK, id), below = (1u << lane) - 1u;
    unsigned rest = id >= 0 ? grp & ~below & ~(1u << lane) : 0u;  // the group's later lanes
    const bool first = id >= 0 && (grp & below) == 0;
    int pos = __popc(grp & below);
    while (__any_sync(HP_FULL_MASK, rest != 0)) {
        const int next = rest ? __ffs(rest) - 1 : lane;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const float o = __shfl_sync(HP_FULL_MASK, x[k], next);
            if (rest) x[k] += o;
        }
        rest &= __ballot_sync(HP_FULL_MASK, !(pos & 1));
        pos >>= 1;
    }
    return first;
}

__global__ void __launch_bounds__(AB) k_adjoint(const float* __restrict__ verts, int64_t nv,
                                                const int32_t* __restrict__ tris, int64_t ntri,
                                                const float4* __restrict__ rays,
                                                const int4* __restrict__ results,
                                                const float* __restrict__ dl, int64_t num_rays,
                                                float* __restrict__ dverts, bool dense, int* err) {
    const int64_t i = blockIdx.x * (int64_t)AB + threadIdx.x;
    int hit = -1;  // triangle of the lane's contribution
    int idx[3] = {0, 0, 0};
    float g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (i < num_rays) {
        const int4 res = results[i];
        const int tri = res.x;
        if (tri >= 0 && tri < ntri) {
            const float u = __int_as_float(res.z), v = __int_as_float(res.w);
            uint32_t l[3];
            load3(reinterpret_cast<const uint32_t*>(dl + 3 * i), l[0], l[1], l[2]);
            const float gt = __uint_as_float(l[0]), gu = __uint_as_float(l[1]), gv = __uint_as_float(l[2]);
            const float4 d4 = rays[2 * i + 1];
            load3(reinterpret_cast<const uint32_t*>(tris + 3 * (int64_t)tri), l[0], l[1], l[2]);
            float3 p[3];
            bool ok = true;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                idx[k] = (int)l[k];
                if (idx[k] < 0 || idx[k] >= nv) { ok = false; idx[k] = 0; }
                load_vertex(verts, nv, idx[k], p[k].x, p[k].y, p[k].z, err, tri);
            }
            if (!ok) hp_report(err, HP_DEV_BAD_INPUT, tri);
            const float3 a = make_float3(p[0].x - p[2].x, p[0].y - p[2].y, p[0].z - p[2].z);
            const float3 b = make_float3(p[1].x - p[2].x, p[1].y - p[2].y, p[1].z - p[2].z);
            const float3 c = make_float3(-d4.x, -d4.y, -d4.z);
            const float3 bc = cross3(b, c), ca = cross3(c, a), ab = cross3(a, b);
            const float det = dot3(a, bc);
            if (ok && det != 0.0f) {
                const float qx = __fdiv_rn(comb3(gu, bc.x, gv, ca.x, gt, ab.x), det);
                const float qy = __fdiv_rn(comb3(gu, bc.y, gv, ca.y, gt, ab.y), det);
                const float qz = __fdiv_rn(comb3(gu, bc.z, gv, ca.z, gt, ab.z), det);
                const float w[3] = {u, v, __fsub_rn(__fsub_rn(1.0f, u), v)};
                hit = tri;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    g[3 * k] = -__fmul_rn(w[k], qx);
                    g[3 * k + 1] = -__fmul_rn(w[k], qy);
                    g[3 * k + 2] = -__fmul_rn(w[k], qz);
                }
            }
        }
    }
    // Lanes of one triangle sum their nine components first; then, corner by corner, the
    // triangles' first lanes with the same vertex sum its three, lest they add to one
    // address one after another: where the warp's first triangle shares its vertex with two
    // others (on a fan of 4,096 triangles around a vertex 4.2 M rays take 12.8 ms without,
    // 0.44 with), and everywhere on a mesh so coarse that warps queue for its vertices
    // (`dense`; 2 x 4 x 4 triangles 5.25 and 3.46 ms, 2 x 32 x 32 equal). Elsewhere the search
    // costs more than it saves: a 1 M-triangle heightfield, where two share, 0.134 ms with it,
    // 0.092 without.
    const bool lead = join(hit, g);
    const unsigned leads = __ballot_sync(HP_FULL_MASK, lead);
    if (leads == 0) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int front = __shfl_sync(HP_FULL_MASK, idx[k], __ffs(leads) - 1);
        bool add = lead;
        float v[3] = {g[3 * k], g[3 * k + 1], g[3 * k + 2]};
        const int same = __popc(__ballot_sync(HP_FULL_MASK, lead && idx[k] == front));
        if (dense || same >= 3) add = join(lead ? idx[k] : -1, v);
        if (add) add3(dverts, idx[k], v[0], v[1], v[2]);
    }
}

// One thread per leaf node: re-woopify its triangles, store its box, then
// climb through parent links; the second child to arrive at a node finishes it.
__global__ void __launch_bounds__(AB) k_refit(const float* __restrict__ verts, int64_t nv,
                                              const int32_t* __restrict__ tris,
                                              const int32_t* __restrict__ tri_idx,
                                              hp_node_bin* nodes, float4* __restrict__ woop,
                                              int* counters, const hp_bvh_info* info, int n_refs,
                                              int* err) {
    const int num_int = info->num_interior, num_leaf = info->num_leaf;
    const int li = blockIdx.x * AB + threadIdx.x;
    if (li >= num_leaf) return;
    const int leaf = num_int + li;
    const int4 meta = nodes[leaf].meta;
    if (meta.x < 0 || meta.y > n_refs || meta.x > meta.y) {
        hp_report(err, HP_DEV_BAD_INDEX, leaf);
        return;
    }
    float mn[3] = {HP_MAX_FLOAT, HP_MAX_FLOAT, HP_MAX_FLOAT};
    float mx[3] = {-HP_MAX_FLOAT, -HP_MAX_FLOAT, -HP_MAX_FLOAT};
    for (int r = meta.x; r < meta.y; ++r) {
        const tri_verts t = load_tri<true>(verts, nv, tris, tri_idx[r], err);
        mn[0] = fminf(mn[0], fminf(fminf(t.x0, t.x1), t.x2));
        mn[1] = fminf(mn[1], fminf(fminf(t.y0, t.y1), t.y2));
        mn[2] = fminf(mn[2], fminf(fminf(t.z0, t.z1), t.z2));
        mx[0] = fmaxf(mx[0], fmaxf(fmaxf(t.x0, t.x1), t.x2));
        mx[1] = fmaxf(mx[1], fmaxf(fmaxf(t.y0, t.y1), t.y2));
        mx[2] = fmaxf(mx[2], fmaxf(fmaxf(t.z0, t.z1), t.z2));
        float4 w0, w1, w2;
        hp_woop(t.x0, t.y0, t.z0, t.x1, t.y1, t.z1, t.x2, t.y2, t.z2, w0, w1, w2);
        woop[3 * (int64_t)r] = w0;
        woop[3 * (int64_t)r + 1] = w1;
        woop[3 * (int64_t)r + 2] = w2;
    }
    if (meta.x >= meta.y) return;  // empty leaf (single-triangle BVH): keeps its inverted box
    float4 bmn = make_float4(mn[0], mn[1], mn[2], 0.0f), bmx = make_float4(mx[0], mx[1], mx[2], 0.0f);
    nodes[leaf].c0xy = make_float4(bmn.x, bmx.x, bmn.y, bmx.y);
    nodes[leaf].c1xy = make_float4(bmn.x, bmx.x, bmn.y, bmx.y);
    nodes[leaf].cz = make_float4(bmn.z, bmx.z, bmn.z, bmx.z);
    int child = leaf;
    int node = meta.w;
    int guard = 0;
    int4 pm = node >= 0 && node < num_int ? __ldcg(&nodes[node].meta) : make_int4(0, 0, 0, -1);
    while (node >= 0) {
        if (node >= num_int || ++guard > num_int) {
            hp_report(err, HP_DEV_BAD_INDEX, node);
            return;
        }
        hp_node_bin* pn = nodes + node;
        const bool first = (pm.x < 0 ? ~pm.x : pm.x) == child;
        if (first) {
            __stcg(&pn->c0xy, make_float4(bmn.x, bmx.x, bmn.y, bmx.y));
            __stcg(reinterpret_cast<float2*>(&pn->cz), make_float2(bmn.z, bmx.z));
        } else {
            __stcg(&pn->c1xy, make_float4(bmn.x, bmx.x, bmn.y, bmx.y));
            __stcg(reinterpret_cast<float2*>(&pn->cz) + 1, make_float2(bmn.z, bmx.z));
        }
        // The parent's links are read while the arrival travels; a refit changes
        // no link.
        const int up = pm.w;
        const int4 um = up >= 0 && up < num_int ? __ldcg(&nodes[up].meta) : make_int4(0, 0, 0, -1);
        if (hp_arrive(&counters[node]) == 0) return;
        // the second to arrive has its own box and reads the other child's
        const float4 o = __ldcg(first ? &pn->c1xy : &pn->c0xy);
        const float2 oz = __ldcg(reinterpret_cast<const float2*>(&pn->cz) + (first ? 1 : 0));
        bmn = make_float4(fminf(bmn.x, o.x), fminf(bmn.y, o.z), fminf(bmn.z, oz.x), 0.0f);
        bmx = make_float4(fmaxf(bmx.x, o.y), fmaxf(bmx.y, o.w), fmaxf(bmx.z, oz.y), 0.0f);
        child = node;
        node = up;
        pm = um;
    }
}

}  // namespace

hp_status hp_adjoint_launch(hp_ctx* ctx, const hp_mesh* m, const float* rays, const int32_t* results,
                            const float* dl_dtuv, int64_t num_rays, float* dl_dvertices,
                            cudaStream_t s) {
    if (num_rays <= 0) return HP_OK;
    k_adjoint<<<hp_div_up(num_rays, AB), AB, 0, s>>>(
        m->vertices, m->num_vertices, m->triangles, m->num_triangles,
        reinterpret_cast<const float4*>(rays), reinterpret_cast<const int4*>(results), dl_dtuv,
        num_rays, dl_dvertices, num_rays / 2048 >= m->num_vertices, ctx->d_status);
    HP_CUDA(cudaGetLastError());
    hp_count_launch();
    hp_mark(ctx, s, "adjoint");
    return HP_OK;
}

hp_status hp_refit_launch(hp_ctx* ctx, hp_bvh_impl* b, int64_t n_refs, const hp_mesh* m,
                          cudaStream_t s) {
    if (n_refs <= 0) return HP_OK;
    HP_CUDA(cudaMemsetAsync(b->counters, 0, sizeof(int) * std::max<int64_t>(n_refs, 2), s));
    const int64_t max_leaves = std::max<int64_t>(n_refs, 2);
    k_refit<<<hp_div_up(max_leaves, AB), AB, 0, s>>>(m->vertices, m->num_vertices, m->triangles,
                                                     b->tri_idx, b->nodes, b->woop, b->counters,
                                                     b->info, (int)n_refs, ctx->d_status);
    HP_CUDA(cudaGetLastError());
    hp_count_launch();
    hp_mark(ctx, s, "refit");
    return HP_OK;
}
