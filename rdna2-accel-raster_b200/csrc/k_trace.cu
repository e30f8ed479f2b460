// k_trace.cu — ray traversal kernels.
//
//  k_trace4   the engine's 4-wide traversal (rq_trace, trace_engine.cuh) over
//             a ray buffer.  Closest hit: nearest child first (ties by slot);
//             any hit: by slot, to the first accepted triangle.  Watertight
//             or Moller-Trumbore triangles.
//  k_trace_radv  the same order over a RADV image (Box32 + triangle nodes).
//  k_ref4     software_bvh_bvh4.comp:96-195 as published (24-entry stack that
//             drops overflow, leaves tested inline far-to-near, RayStats).
//  k_ref2     software_bvh_lds.comp:86-175 as published (hitFound flag).
#include "rq_device.cuh"
#include "rq_internal.h"
#include "trace_engine.cuh"

namespace {

constexpr int kT = 128;
// rq_trace's engine: idle lanes are refilled once half the warp is idle, and
// 8 blocks of kT threads share an SM (64 registers).  Measured on B200 over
// 2^20 procedural rays, coherent and incoherent, at 968 / 99,458 / 999,698
// triangles: 8-18 % faster than refilling every idle lane at once with no
// register cap at five of the six points, equal at the sixth (968
// triangles, incoherent).
constexpr int kTraceRefill = 16;
constexpr int kTraceBlocksPerSm = 8;
constexpr uint32_t kSmallTree = 4096, kLargeTree = 1u << 17;  // 4-wide nodes

__device__ __forceinline__ void store_miss(rq_hit* hits, uint32_t i) {
    reinterpret_cast<uint4*>(hits)[i] = make_uint4(0u, __float_as_uint(-1.0f), 0xffffffffu, 0xffffffffu);
}

// Ray source of rq_trace: rays from a buffer, hits to a buffer.
template <bool STATS, bool BARY>
struct BufSrc {
    struct Meta {};
    uint32_t total;
    const rq_ray* rays;
    const uint32_t* perm;
    rq_hit* hits;
    float* bary;
    rq_ray_stats* stats;

    __device__ bool make(uint32_t id, rq::Ray& r, Meta&) const {
        const float4* rp = reinterpret_cast<const float4*>(rays + id);
        const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
        r.o = rq::F3{r0.x, r0.y, r0.z};
        r.d = rq::F3{r1.x, r1.y, r1.z};
        r.tmin = r0.w;
        r.tmax = r1.w;
        return true;
    }

    __device__ void finish(uint32_t id, const Meta&, const rq::Ray&, const rq::Hit& h) const {
        if (h.hit) {
            const uint32_t pid = perm ? __ldg(perm + h.idx) : h.idx;
            reinterpret_cast<uint4*>(hits)[id] = make_uint4(1u, __float_as_uint(h.t), 0u, pid);
        } else {
            store_miss(hits, id);
        }
        if (BARY) reinterpret_cast<float2*>(bary)[id] = h.hit ? make_float2(h.u, h.v) : make_float2(0.f, 0.f);
        if (STATS) reinterpret_cast<uint4*>(stats)[id] = make_uint4(h.hit ? 1u : 0u, h.boxes, h.tris, 0u);
    }
};

// `max_depth`: levels the stack's `rows` entries cover.  lanes: rays that share a warp.
// few: trace_persistent's.
template <bool ANY, bool MT, bool STATS, bool BARY, bool WIDE>
__global__ void __launch_bounds__(kT, kTraceBlocksPerSm) k_trace4(const rq_bvh4_node* __restrict__ nodes,
                                               const rq_triangle* __restrict__ tris,
                                               const __grid_constant__ BufSrc<STATS, BARY> src,
                                               const uint32_t* __restrict__ counts, uint32_t* ctr, uint32_t* err,
                                               int rows, uint32_t max_depth, uint32_t lanes, int few) {
    extern __shared__ __align__(16) char s_stack[];
    // the rows were picked from the host's copy of the depth; the live depth
    // (after an in-place rebuild) must still fit
    if (blockIdx.x == 0 && threadIdx.x == 0 && __ldg(counts + 2) > max_depth) rq::set_err(err, RQ_DERR_STACK);
    rq::check_leaves(counts, err);
    using Entry = typename rq::OpenNode<ANY, WIDE>::Entry;
    rq::trace_persistent<ANY, MT, STATS, kT, const BufSrc<STATS, BARY>, 32, WIDE>(
        nodes, tris, src, ctr, reinterpret_cast<Entry*>(s_stack) + threadIdx.x, rows, err,
        lanes == 32u ? kTraceRefill : 1, lanes, few);
}

// One ray per thread over a RADV image.  Open nodes as in trace_engine.cuh: one
// stack entry per open box node, its id and the order of the children left; the
// nearest child's id is at hand when its node has been opened, the others' are
// read when their turn comes.  Few rays make a launch of one partial wave (the
// fast builder's use: 16,384 rays on 4,096 triangles), where the time is that
// of a warp's longest union of node chains; such a launch takes every second
// or fourth lane only, so fewer rays share a warp.  24.0 us before (stack of
// children, one loop for boxes and triangles), 21.6 us with full warps, 19.2
// at 16 rays per warp, 18.3 at 8, 18.4 at 4.
constexpr uint32_t kRadvSpread = 2;   // at least 8 rays per warp
constexpr uint32_t kRadvFill = 768;   // threads per SM such a launch may take
// Open nodes that a ray may leave behind it.  This builder's trees are complete
// (2^25 triangles: 14 deep), but any image may come in: a stack of 64 children,
// the form before, held a chain of 63 two-child nodes, so as many rows hold all
// it held.  An entry is 32 bits, a box node's offset (23 bits of 64 bytes) over
// the order of its children left; images past 512 MiB (WIDE) take the order's
// first child in the id's type bits and the others in a byte beside them.
constexpr int kRadvRows = 64;
constexpr uint64_t kRadvNarrow = uint64_t(64) << 23;

template <bool ANY, bool MT, bool BARY, bool WIDE>
__global__ void __launch_bounds__(kT) k_trace_radv(const uint8_t* __restrict__ img, const rq_ray* __restrict__ rays,
                                                   uint32_t n, uint32_t spread, rq_hit* __restrict__ hits,
                                                   float* __restrict__ bary, uint32_t* err) {
    __shared__ uint32_t s_stack[kRadvRows * kT];
    __shared__ uint8_t s_more[WIDE ? kRadvRows * kT : 1];
    const uint32_t g = blockIdx.x * kT + threadIdx.x, i = g >> spread;
    if (i >= n || (g & ((1u << spread) - 1u))) return;
    uint32_t* stk = s_stack + threadIdx.x;
    uint8_t* more = s_more + (WIDE ? threadIdx.x : 0u);
    const uint8_t* base = img + RQ_RADV_BVH_OFFSET;
    const float4* rp = reinterpret_cast<const float4*>(rays + i);
    float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    rq::F3 o{r0.x, r0.y, r0.z}, d{r1.x, r1.y, r1.z};
    const float tmin = r0.w;
    float best = r1.w;
    rq::SlabRay sr;
    sr.ix = rq::safe_inv(d.x);
    sr.iy = rq::safe_inv(d.y);
    sr.iz = rq::safe_inv(d.z);
    sr.ox = o.x * sr.ix;
    sr.oy = o.y * sr.iy;
    sr.oz = o.z * sr.iz;
    rq::WtRay w;
    if (!MT) w = rq::wt_setup(d);
    uint32_t hit_id = 0xffffffffu;
    bool found = false;
    float hu = 0.0f, hv = 0.0f;
    auto node = [&](uint32_t id) { return base + (size_t(id & ~7u) << 3); };
    uint32_t cur = RQ_RADV_NODE_BOX32;  // the node to visit (the root)
    uint32_t top = 0, left = 0;         // the deepest open node, its children left
    int sp = 0;
    auto next = [&]() {
        if (left == 0u) {
            if (sp == 0) return false;
            const uint32_t e = stk[(--sp) * kT];
            top = WIDE ? e : e >> 6;  // (node() drops the lowest three bits)
            left = WIDE ? (e & 7u) | uint32_t(more[sp * kT]) << 3 : e & 511u;
        }
        cur = __ldg(reinterpret_cast<const uint32_t*>(node(top)) + (left & 3u));
        left >>= 3;
        return true;
    };
    for (;;) {
        bool have = true;
        // box nodes, then triangles: a warp's lanes stay in one of the two
        while (have && (cur & 7u) == RQ_RADV_NODE_BOX32) {
            const float4* np = reinterpret_cast<const float4*>(node(cur));
            const uint4 ch = __ldg(reinterpret_cast<const uint4*>(np));
            float cf[24];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                float4 v = rq::ldg4(np + 1 + q);
                cf[4 * q] = v.x;
                cf[4 * q + 1] = v.y;
                cf[4 * q + 2] = v.z;
                cf[4 * q + 3] = v.w;
            }
            const uint32_t ac[4] = {ch.x, ch.y, ch.z, ch.w};
            float tk[4];
            uint32_t hitm = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (rq::slab(sr, tmin, best, cf[6 * k], cf[6 * k + 3], cf[6 * k + 1], cf[6 * k + 4], cf[6 * k + 2],
                             cf[6 * k + 5], tk[k]) &&
                    ac[k] != RQ_RADV_INVALID_NODE)
                    hitm |= 1u << k;
            if (hitm) {
                const uint32_t seq = rq::child_sequence<false>(hitm, tk, !ANY), first = seq & 3u;
                if (seq >> 3) {
                    if (left) {
                        if (sp < kRadvRows) {
                            if (WIDE) more[sp * kT] = uint8_t(left >> 3);
                            stk[(sp++) * kT] = WIDE ? (top & ~7u) | (left & 7u) : (top >> 3) << 9 | left;
                        } else {
                            rq::set_err(err, RQ_DERR_STACK);
                        }
                    }
                    top = cur;
                    left = seq >> 3;
                }
                cur = first < 2u ? (first == 0u ? ac[0] : ac[1]) : (first == 2u ? ac[2] : ac[3]);
            } else {
                have = next();
            }
        }
        bool done = false;
        while (have && (cur & 7u) != RQ_RADV_NODE_BOX32) {
            if ((cur & 7u) != RQ_RADV_NODE_TRIANGLE) {  // (no other type is built)
                have = next();
                continue;
            }
            const float4* np = reinterpret_cast<const float4*>(node(cur));
            float4 a = rq::ldg4(np), b = rq::ldg4(np + 1), c = rq::ldg4(np + 2);
            rq::F3 v0{a.x, a.y, a.z}, v1{a.w, b.x, b.y}, v2{b.z, b.w, c.x};
            float t, u, v;
            bool ok = MT ? rq::mt_test(o, d, v0, v1, v2, 1e-7f, t, u, v) : rq::wt_test(w, o, v0, v1, v2, t, u, v);
            if (ok && t >= tmin && t < best) {
                best = t;
                hit_id = __float_as_uint(__ldg(reinterpret_cast<const float*>(np + 3)));  // triangle_id at byte 48
                found = true;
                hu = u;
                hv = v;
                done = ANY;
                if (ANY) break;
            }
            have = next();
        }
        if (!have || done) break;
    }
    if (found) {
        reinterpret_cast<uint4*>(hits)[i] = make_uint4(1u, __float_as_uint(best), 0u, hit_id);
    } else {
        store_miss(hits, i);
    }
    if (BARY) reinterpret_cast<float2*>(bary)[i] = found ? make_float2(hu, hv) : make_float2(0.f, 0.f);
}

__global__ void __launch_bounds__(kT) k_ref4(const rq_bvh4_node* __restrict__ nodes,
                                             const rq_triangle* __restrict__ tris, const rq_ray* __restrict__ rays,
                                             uint32_t n, rq_ray_stats* __restrict__ stats, rq_hit* __restrict__ hits) {
    __shared__ int32_t s_stack[24 * kT];
    const uint32_t idx = blockIdx.x * kT + threadIdx.x;
    if (idx >= n) return;
    int32_t* stk = s_stack + threadIdx.x;
    const rq_ray r = rays[idx];
    rq::F3 o{r.org[0], r.org[1], r.org[2]}, d{r.dir[0], r.dir[1], r.dir[2]};
    rq::F3 inv{fabsf(d.x) > 1e-6f ? 1.0f / d.x : 1e6f, fabsf(d.y) > 1e-6f ? 1.0f / d.y : 1e6f,
               fabsf(d.z) > 1e-6f ? 1.0f / d.z : 1e6f};
    const float tmin = r.tmin;
    float hitT = r.tmax;
    int hitPrim = -1;
    uint32_t boxTests = 0, triTests = 0;
    stk[0] = 0;
    int ptr = 1;
    while (ptr > 0) {
        const rq_bvh4_node nd = nodes[stk[(--ptr) * kT]];
        boxTests += 4;
        float tEntry[4], tExit[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float t0x = (nd.min_x[k] - o.x) * inv.x, t1x = (nd.max_x[k] - o.x) * inv.x;
            float t0y = (nd.min_y[k] - o.y) * inv.y, t1y = (nd.max_y[k] - o.y) * inv.y;
            float t0z = (nd.min_z[k] - o.z) * inv.z, t1z = (nd.max_z[k] - o.z) * inv.z;
            tEntry[k] = fmaxf(fmaxf(fminf(t0x, t1x), fminf(t0y, t1y)), fmaxf(fminf(t0z, t1z), tmin));
            tExit[k] = fminf(fminf(fmaxf(t0x, t1x), fmaxf(t0y, t1y)), fminf(fmaxf(t0z, t1z), hitT));
        }
        int slot[4];
        float ht[4];
        int hc = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (nd.child_count[k] != 0 && tExit[k] >= tEntry[k]) {
                slot[hc] = k;
                ht[hc] = tEntry[k];
                ++hc;
            }
        if (hc == 0) continue;
        for (int a = 0; a < hc - 1; ++a)
            for (int b = a + 1; b < hc; ++b)
                if (ht[a] < ht[b]) {
                    float tt = ht[a];
                    ht[a] = ht[b];
                    ht[b] = tt;
                    int ts = slot[a];
                    slot[a] = slot[b];
                    slot[b] = ts;
                }
        for (int a = 0; a < hc; ++a) {
            int k = slot[a];
            if (nd.child_count[k] > 0) {
                uint32_t first = uint32_t(~nd.child_index[k]);
                uint32_t cnt = uint32_t(nd.child_count[k]);
                triTests += cnt;
                for (uint32_t p = 0; p < cnt; ++p) {
                    const rq_triangle tr = tris[first + p];
                    rq::F3 v0{tr.v0[0], tr.v0[1], tr.v0[2]}, v1{tr.v1[0], tr.v1[1], tr.v1[2]},
                        v2{tr.v2[0], tr.v2[1], tr.v2[2]};
                    float t, u, v;
                    if (!rq::mt_test(o, d, v0, v1, v2, 1e-7f, t, u, v)) continue;
                    if (t >= tmin && t < hitT) {
                        hitT = t;
                        hitPrim = int(first + p);
                    }
                }
            } else if (nd.child_count[k] < 0) {
                if (ptr < 24) stk[(ptr++) * kT] = nd.child_index[k];
            }
        }
    }
    if (stats) reinterpret_cast<uint4*>(stats)[idx] = make_uint4(hitPrim >= 0 ? 1u : 0u, boxTests, triTests, 0u);
    if (hits) {
        if (hitPrim >= 0)
            reinterpret_cast<uint4*>(hits)[idx] = make_uint4(1u, __float_as_uint(hitT), 0u, uint32_t(hitPrim));
        else
            store_miss(hits, idx);
    }
}

__device__ __forceinline__ bool ref2_box(const rq_bvh2_node& nd, rq::F3 o, rq::F3 inv, float closestT, float& tb) {
    float t0x = (nd.aabb_min[0] - o.x) * inv.x, t1x = (nd.aabb_max[0] - o.x) * inv.x;
    float t0y = (nd.aabb_min[1] - o.y) * inv.y, t1y = (nd.aabb_max[1] - o.y) * inv.y;
    float t0z = (nd.aabb_min[2] - o.z) * inv.z, t1z = (nd.aabb_max[2] - o.z) * inv.z;
    float tNear = fmaxf(fmaxf(fminf(t0x, t1x), fminf(t0y, t1y)), fminf(t0z, t1z));
    float tFar = fminf(fminf(fmaxf(t0x, t1x), fmaxf(t0y, t1y)), fmaxf(t0z, t1z));
    tb = tNear;
    return (tFar >= fmaxf(0.0f, tNear)) && (tNear < closestT);
}

__device__ __forceinline__ float ref2_clamp(float x) { return fabsf(x) > 1e-8f ? x : (x >= 0.0f ? 1e-8f : -1e-8f); }

__global__ void __launch_bounds__(kT) k_ref2(const rq_bvh2_node* __restrict__ nodes,
                                             const rq_triangle* __restrict__ tris, const rq_ray* __restrict__ rays,
                                             uint32_t n, float t_eps, uint32_t* __restrict__ flags) {
    __shared__ uint32_t s_stack[32 * kT];
    const uint32_t idx = blockIdx.x * kT + threadIdx.x;
    if (idx >= n) return;
    uint32_t* stk = s_stack + threadIdx.x;
    const rq_ray r = rays[idx];
    rq::F3 o{r.org[0], r.org[1], r.org[2]}, d{r.dir[0], r.dir[1], r.dir[2]};
    rq::F3 inv{1.0f / ref2_clamp(d.x), 1.0f / ref2_clamp(d.y), 1.0f / ref2_clamp(d.z)};
    float closestT = r.tmax;
    uint32_t hitFound = 0;
    int sp = 0;
    stk[(sp++) * kT] = 0;
    while (sp > 0) {
        const rq_bvh2_node nd = nodes[stk[(--sp) * kT]];
        float tb;
        if (!ref2_box(nd, o, inv, closestT, tb)) continue;
        if (nd.left_child < 0) {
            uint32_t start = uint32_t(~nd.left_child);
            for (int32_t q = 0; q < nd.right_child; ++q) {
                const rq_triangle tr = tris[start + uint32_t(q)];
                rq::F3 v0{tr.v0[0], tr.v0[1], tr.v0[2]}, v1{tr.v1[0], tr.v1[1], tr.v1[2]},
                    v2{tr.v2[0], tr.v2[1], tr.v2[2]};
                float t, u, v;
                if (!rq::mt_test(o, d, v0, v1, v2, 1e-8f, t, u, v)) continue;
                if (t > t_eps && t < closestT) {
                    closestT = t;
                    hitFound = 1;
                }
            }
        } else {
            uint32_t l = uint32_t(nd.left_child), rr = uint32_t(nd.right_child);
            float tl, tr;
            bool hl = ref2_box(nodes[l], o, inv, closestT, tl), hr = ref2_box(nodes[rr], o, inv, closestT, tr);
            if (hl && hr) {
                if (tl < tr) {
                    if (sp < 32) stk[(sp++) * kT] = rr;
                    if (sp < 32) stk[(sp++) * kT] = l;
                } else {
                    if (sp < 32) stk[(sp++) * kT] = l;
                    if (sp < 32) stk[(sp++) * kT] = rr;
                }
            } else if (hl) {
                if (sp < 32) stk[(sp++) * kT] = l;
            } else if (hr) {
                if (sp < 32) stk[(sp++) * kT] = rr;
            }
        }
    }
    flags[idx] = hitFound;
}

template <bool ANY, bool MT, bool EX>
cudaError_t launch4(rq_ctx* ctx, const rq_bvh* b, const rq_ray* rays, uint32_t n, rq_hit* hits, float* bary,
                    rq_ray_stats* stats, cudaStream_t st) {
    // Stack rows (an entry per open node of a path) by the depth the host
    // knows, with room for the levels an in-place rebuild may add.  At most
    // 44 rows of 4 or 8 bytes: kTraceBlocksPerSm blocks always fit an SM
    // (64 registers, 45 KB at most with the 8-byte entries of 4 blocks).
    const uint32_t d = b->h_counts[2];
    const uint32_t max_depth = d <= 8u ? 10u : (d <= 19u ? 21u : 42u);
    const bool wide = !ANY && b->cap_nodes4 > RQ_NARROW_NODES;
    auto kern = wide ? k_trace4<ANY, MT, EX, EX, !ANY> : k_trace4<ANY, MT, EX, EX, false>;
    const int rows = int(max_depth) + 2;
    const size_t smem = size_t(rows) * kT * (wide ? 8 : 4);
    // persistent grid: every SM filled, never more blocks than there are chunks
    uint32_t blocks = uint32_t(ctx->num_sms) * uint32_t(wide && rows > 24 ? 4 : kTraceBlocksPerSm);
    // A batch of less than one ray per resident lane takes the time of its
    // slowest warp, whose length grows with the rays that share it: it is
    // spread over all the warps there are, at 4, 8 or 16 rays each, but not down
    // to a ray for every lane that takes part: a warp that starts full has no
    // slack, and the next step is as fast or faster from 3/4 on, on trees of more
    // than kLargeTree nodes, whose walks differ more, from 7/8 on.  Closest hit,
    // us at 4 / 8 / 16 / 32 rays (4 and 8 hold 18,944 and 37,888 rays):
    //               99,458 triangles            999,698
    //   12,000      44.8 / 44.7 / 46.5 / 48.6   48.8 / 48.8 / 50.6 / 53.5
    //   18,000      50.8 / 48.8 / 48.7 / 51.0   53.5 / 51.7 / 50.9 / 55.2
    //   37,000        -  / 55.0 / 55.1 / 54.6     -  / 61.0 / 57.2 / 57.7
    //   65,536        -  /   -  / 61.2 / 59.3     -  /   -  / 65.2 / 65.3
    // (any hit, 65,536 rays on 999,698: 58.1 at 16, 60.5 at 32; 8.3M triangles,
    // closest hit 87.0 and 90.3; 968 triangles 42.9 and 40.5).
    const uint32_t warps = blocks * (kT / 32);
    const uint32_t eighths = b->h_counts[1] > kLargeTree ? 7 : 6;
    uint32_t lanes = 4;
    while (lanes < 32u && n > lanes * warps / 8u * eighths) lanes *= 2;
    // On small trees a node phase is a few steps, and leaving it early costs more
    // than the idle lanes do (2^20 rays, us with and without: 968 triangles
    // incoherent 166 / 156, coherent 101 / 98, 8,192 coherent 113 / 110; 99,458
    // equal; 999,698 incoherent 419 / 432).
    const int few = b->h_counts[1] <= kSmallTree ? 0 : rq::kFewSearch;
    const uint32_t need = (n + (kT / 32) * lanes - 1) / ((kT / 32) * lanes);
    if (blocks > need) blocks = need;
    BufSrc<EX, EX> src;
    src.total = n;
    src.rays = rays;
    src.perm = b->perm;
    src.hits = hits;
    src.bary = bary;
    src.stats = stats;
    cudaError_t e = cudaMemsetAsync(ctx->d_ctr, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    kern<<<blocks, kT, smem, st>>>(b->nodes4, b->tris, src, b->d_counts, ctx->d_ctr, ctx->d_err, rows, max_depth,
                                   lanes, few);
    return cudaGetLastError();
}

template <bool ANY, bool MT>
cudaError_t launch4_opts(bool ex, rq_ctx* ctx, const rq_bvh* b, const rq_ray* rays, uint32_t n, rq_hit* hits,
                         float* bary, rq_ray_stats* stats, cudaStream_t st) {
    if (ex) return launch4<ANY, MT, true>(ctx, b, rays, n, hits, bary, stats, st);
    return launch4<ANY, MT, false>(ctx, b, rays, n, hits, bary, stats, st);
}

}  // namespace

int rq_launch_trace(rq_ctx* ctx, const rq_bvh* bvh, const rq_ray* rays, uint32_t n, uint32_t flags, rq_hit* hits,
                    float* bary, rq_ray_stats* stats, cudaStream_t st) {
    if (n == 0) return RQ_OK;
    if (3u * bvh->h_counts[2] + 1u > 128u)
        return rq_set_error(ctx, RQ_ERR_UNSUPPORTED, "4-wide tree deeper than 42 levels");
    // With stats or barycentrics requested, the kernel variant that records
    // both is used; a null destination gets a scratch sink.
    rq_ray_stats* st_out = stats;
    float* ba_out = bary;
    if ((stats != nullptr) != (bary != nullptr)) {
        size_t need = size_t(n) * (stats ? 8 : 16);
        int rc = rq_ensure_scratch(ctx, need, st);
        if (rc) return rc;
        if (!stats) st_out = static_cast<rq_ray_stats*>(ctx->scratch);
        if (!bary) ba_out = static_cast<float*>(ctx->scratch);
    }
    const bool any = flags & RQ_TRACE_ANY, mt = flags & RQ_TRI_MT;
    const bool ex = stats || bary;
    cudaError_t e;
    if (any && mt)
        e = launch4_opts<true, true>(ex, ctx, bvh, rays, n, hits, ba_out, st_out, st);
    else if (any)
        e = launch4_opts<true, false>(ex, ctx, bvh, rays, n, hits, ba_out, st_out, st);
    else if (mt)
        e = launch4_opts<false, true>(ex, ctx, bvh, rays, n, hits, ba_out, st_out, st);
    else
        e = launch4_opts<false, false>(ex, ctx, bvh, rays, n, hits, ba_out, st_out, st);
    return rq_cuda_status(ctx, e, "trace launch");
}

int rq_launch_trace_ref4(rq_ctx* ctx, const rq_bvh4_node* nodes, const rq_triangle* tris, const rq_ray* rays,
                         uint32_t n, rq_ray_stats* stats, rq_hit* hits, cudaStream_t st) {
    if (n == 0) return RQ_OK;
    k_ref4<<<(n + kT - 1) / kT, kT, 0, st>>>(nodes, tris, rays, n, stats, hits);
    return rq_cuda_status(ctx, cudaGetLastError(), "reference bvh4 trace launch");
}

int rq_launch_trace_ref2(rq_ctx* ctx, const rq_bvh2_node* nodes, const rq_triangle* tris, const rq_ray* rays,
                         uint32_t n, float t_eps, uint32_t* flags, cudaStream_t st) {
    if (n == 0) return RQ_OK;
    k_ref2<<<(n + kT - 1) / kT, kT, 0, st>>>(nodes, tris, rays, n, t_eps, flags);
    return rq_cuda_status(ctx, cudaGetLastError(), "reference bvh2 trace launch");
}

int rq_launch_trace_radv(rq_ctx* ctx, const void* img, uint64_t bytes, const rq_ray* rays, uint32_t n,
                         uint32_t flags, rq_hit* hits, float* bary, cudaStream_t st) {
    if (n == 0) return RQ_OK;
    const uint8_t* im = static_cast<const uint8_t*>(img);
    const bool any = flags & RQ_TRACE_ANY, mt = flags & RQ_TRI_MT, b = bary != nullptr;
    // fewer rays per warp while that still leaves one wave
    uint32_t spread = 0;
    while (spread < kRadvSpread && (uint64_t(n) << (spread + 1)) <= uint64_t(ctx->num_sms) * kRadvFill) ++spread;
    dim3 g(uint32_t(((uint64_t(n) << spread) + kT - 1) / kT));
    const bool wide = bytes > kRadvNarrow;
#define RQ_RADV_CASE(A, M, B)                                                                                 \
    (wide ? k_trace_radv<A, M, B, true> : k_trace_radv<A, M, B, false>)<<<g, kT, 0, st>>>(im, rays, n, spread, \
                                                                                          hits, bary, ctx->d_err)
    if (any && mt && b) RQ_RADV_CASE(true, true, true);
    else if (any && mt) RQ_RADV_CASE(true, true, false);
    else if (any && b) RQ_RADV_CASE(true, false, true);
    else if (any) RQ_RADV_CASE(true, false, false);
    else if (mt && b) RQ_RADV_CASE(false, true, true);
    else if (mt) RQ_RADV_CASE(false, true, false);
    else if (b) RQ_RADV_CASE(false, false, true);
    else RQ_RADV_CASE(false, false, false);
#undef RQ_RADV_CASE
    return rq_cuda_status(ctx, cudaGetLastError(), "radv trace launch");
}
