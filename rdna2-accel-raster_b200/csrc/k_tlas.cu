// k_tlas.cu — two-level scenes: instances of BLAS handles, each with an
// object-to-world transform and an instance id, under a top-level BVH (the
// instance acceleration structures the reference builds through the driver,
// common/vk_bvh.cpp:237-336, with the VkAccelerationStructureInstanceKHR
// records of benchmarks/exp1_visbuf/visbuf_main.cpp:762-771).
//
//  k_instance_boxes  world box of each instance: the BLAS root node's slot
//                    boxes united, its 8 corners transformed, widened by
//                    2^-20 of the coordinate magnitudes (rounding of the
//                    transform must not shrink it); written as the
//                    degenerate triangle (min, max, min), whose bounds are
//                    exactly the box, so the LBVH build of rq_build makes
//                    the top-level tree (one instance per leaf).
//  k_trace_tlas      a ray per lane, idle lanes refilled from the block's.  The
//                    stack holds top-level entries; at an instance leaf the
//                    ray is moved into object space (origin and direction by
//                    the inverse transform, the direction not renormalised,
//                    so t is the same in both spaces and one best-t serves
//                    all instances), a marker entry is pushed and then the
//                    BLAS root; popping the marker returns to world space.
//                    Closest hit sorts children near-to-far at both levels.
//                    The node loop holds box tests alone: triangles, entering
//                    an instance (a matrix, nine divisions) and leaving it
//                    wait until every lane of the warp has such work or none,
//                    so no lane waits for another's in between.
#include <algorithm>

#include "rq_device.cuh"
#include "rq_internal.h"
#include "rq_tlas.h"
#include "trace_engine.cuh"

namespace {

using namespace rq;

constexpr int kTT = 128;
constexpr int kTlasBlocks = 8;   // blocks per SM: 64 registers
constexpr int kTlasRefill = 8;   // idle lanes of a warp that call for new rays (16: 659 us, 24: 765 us)
// A block's rays (its warps take them 32 at a time): an equal share of the
// launch for every block the device holds at once, so there is one wave, but
// at least a ray per lane and at most kTlasMaxRays, so that a large launch
// still evens out over several waves.  No counter is shared between launches:
// launches on several streams do not meet.  518,400 random rays over 256
// instances of 8 meshes: 825 us with a thread per ray and everything in one
// loop, 605 us at 512 rays per block; 128 (a ray per lane, no refill) 913 us,
// 1,024 (fewer blocks than fit) 899 us.
constexpr uint32_t kTlasMaxRays = 2048;
constexpr int32_t kMarker = 0x40000000;  // pending: leave the instance

__global__ void __launch_bounds__(128) k_instance_boxes(const TlasInst* __restrict__ inst,
                                                        const float* __restrict__ fwd, uint32_t n,
                                                        float* __restrict__ tri9) {
    const uint32_t i = blockIdx.x * 128u + threadIdx.x;
    if (i >= n) return;
    const float4* np = reinterpret_cast<const float4*>(inst[i].nodes);
    const float4 mnx = np[0], mxx = np[1], mny = np[2], mxy = np[3], mnz = np[4], mxz = np[5];
    const int4 cnt = reinterpret_cast<const int4*>(np)[7];
    const float amnx[4] = {mnx.x, mnx.y, mnx.z, mnx.w}, amxx[4] = {mxx.x, mxx.y, mxx.z, mxx.w};
    const float amny[4] = {mny.x, mny.y, mny.z, mny.w}, amxy[4] = {mxy.x, mxy.y, mxy.z, mxy.w};
    const float amnz[4] = {mnz.x, mnz.y, mnz.z, mnz.w}, amxz[4] = {mxz.x, mxz.y, mxz.z, mxz.w};
    const int32_t acc[4] = {cnt.x, cnt.y, cnt.z, cnt.w};
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < 4; ++k) {
        if (acc[k] == 0) continue;
        lo[0] = fminf(lo[0], amnx[k]);
        lo[1] = fminf(lo[1], amny[k]);
        lo[2] = fminf(lo[2], amnz[k]);
        hi[0] = fmaxf(hi[0], amxx[k]);
        hi[1] = fmaxf(hi[1], amxy[k]);
        hi[2] = fmaxf(hi[2], amxz[k]);
    }
    const float* f = fwd + 12ull * i;
    float wlo[3] = {INFINITY, INFINITY, INFINITY}, whi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int c = 0; c < 8; ++c) {
        const float x = (c & 1) ? hi[0] : lo[0], y = (c & 2) ? hi[1] : lo[1], z = (c & 4) ? hi[2] : lo[2];
        for (int r = 0; r < 3; ++r) {
            const float w = ((f[4 * r] * x + f[4 * r + 1] * y) + f[4 * r + 2] * z) + f[4 * r + 3];
            wlo[r] = fminf(wlo[r], w);
            whi[r] = fmaxf(whi[r], w);
        }
    }
    float* t = tri9 + 9ull * i;
    for (int r = 0; r < 3; ++r) {
        const float pad = (fabsf(wlo[r]) + fabsf(whi[r])) * 0x1p-20f;
        const float a = wlo[r] - pad, b = whi[r] + pad;
        t[r] = a;
        t[3 + r] = b;
        t[6 + r] = a;
    }
}

__device__ __forceinline__ SlabRay slab_setup(F3 o, F3 d) {
    SlabRay sr;
    sr.ix = safe_inv(d.x);
    sr.iy = safe_inv(d.y);
    sr.iz = safe_inv(d.z);
    sr.ox = o.x * sr.ix;
    sr.oy = o.y * sr.iy;
    sr.oz = o.z * sr.iz;
    return sr;
}

// A lane's pending work outside the node loop: a triangle leaf or an instance
// (entries with bit 31) or the marker that ends an instance.
template <bool ANY, bool MT, bool WIDE>
__global__ void __launch_bounds__(kTT, kTlasBlocks)
    k_trace_tlas(const rq_bvh4_node* __restrict__ top_nodes, const uint32_t* __restrict__ top_perm,
                 const TlasInst* __restrict__ inst, const rq_ray* __restrict__ rays, uint32_t n, uint32_t cull,
                 uint32_t per_block, rq_hit* __restrict__ hits, int rows, uint32_t* err) {
    extern __shared__ __align__(16) char s_stack[];
    using Open = OpenNode<ANY, WIDE>;
    using Entry = typename Open::Entry;
    constexpr Entry kLeave = ~Entry(0);  // "leave the instance": no node's entry (a mask of 15 would need node 2^28 - 1)
    __shared__ uint32_t s_next;  // the block's next ray
    if (threadIdx.x == 0) s_next = blockIdx.x * per_block;
    __syncthreads();
    const uint32_t last = min(n, (blockIdx.x + 1u) * per_block);
    Entry* stk = reinterpret_cast<Entry*>(s_stack) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
    uint32_t next = 0, end = 0;  // the warp's chunk of ray ids
    bool exhausted = false;
    bool active = false;
    uint32_t id = 0;
    float tmin = 0.0f, best = 0.0f;
    SlabRay sr{};
    F3 oo{}, od{};  // the ray in the current space
    WtRay w{};
    const rq_bvh4_node* nodes = top_nodes;
    const TlasInst* in = nullptr;  // the instance the ray is inside, or null
    bool hit = false;
    uint32_t hit_inst = 0, hit_prim = 0;
    int sp = 0;
    Open top;  // the deepest open node
    top.left = 0;
    for (;;) {
        // ---- new rays for idle lanes, once enough are idle
        uint32_t idle = __ballot_sync(kFull, !active);
        const bool go = __popc(idle) >= kTlasRefill || idle == kFull;
        while (go && idle && !exhausted) {
            if (next == end) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(&s_next, 32u);
                base = __shfl_sync(kFull, base, 0);
                if (base >= last) {
                    exhausted = true;
                    break;
                }
                next = base;
                end = min(base + 32u, last);
            }
            const uint32_t take = min(uint32_t(__popc(idle)), end - next);
            const uint32_t rank = __popc(idle & lt_mask);
            if (((idle >> lane) & 1u) && rank < take) {
                id = next + rank;
                const float4* rp = reinterpret_cast<const float4*>(rays + id);
                const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
                sr = slab_setup(F3{r0.x, r0.y, r0.z}, F3{r1.x, r1.y, r1.z});
                tmin = r0.w;
                best = r1.w;
                nodes = top_nodes;
                in = nullptr;
                hit = false;
                top.root();
                sp = 0;
                active = true;
            }
            next += take;
            idle = __ballot_sync(kFull, !active);
        }
        if (!__any_sync(kFull, active)) {
            if (exhausted) break;
            continue;
        }
        // ---- node phase, until every lane holds other work or is done
        int32_t pend = 0;  // a leaf (bit 31 set) or kMarker
        for (;;) {
            const bool want = active && pend == 0 && (top.left != 0u || sp > 0);
            const uint32_t wm = __ballot_sync(kFull, want);
            if (!wm) break;
            if (__popc(wm) <= kFewSearch && __popc(__ballot_sync(kFull, pend != 0)) >= kLeafWait) break;
            if (!want) continue;
            if (top.left == 0u) {
                const Entry e = stk[(--sp) * kTT];
                if (e == kLeave) {
                    pend = kMarker;
                    continue;
                }
                top.unpack(e);
            }
            const uint32_t slot = top.take();
            int32_t ci, cc;
            child_of(nodes, top.node, slot, ci, cc);
            if (cc >= 0) {
                if (cc > 0) pend = int32_t(0x80000000u | (uint32_t(cc - 1) << 27) | uint32_t(~ci));
                continue;
            }
            float tk[4];
            const uint32_t hitm =
                box4_hits<false>(GlobalRows{reinterpret_cast<const float4*>(nodes + ci)}, sr, tmin, best, tk);
            if (hitm) {
                if (top.left) {
                    if (sp < rows)
                        stk[(sp++) * kTT] = top.pack();
                    else
                        set_err(err, RQ_DERR_STACK);
                }
                top.node = ci;
                top.left = ANY ? hitm : child_sequence<false>(hitm, tk, true);
            }
        }
        // ---- the lanes' other work
        bool done = false;
        if (active && pend != 0) {
            const uint32_t first = uint32_t(pend) & 0x07ffffffu;
            if (pend == kMarker) {  // back to the top level
                const float4* rp = reinterpret_cast<const float4*>(rays + id);
                const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
                sr = slab_setup(F3{r0.x, r0.y, r0.z}, F3{r1.x, r1.y, r1.z});
                nodes = top_nodes;
                in = nullptr;
            } else if (!in) {  // an instance (one per top-level leaf)
                const TlasInst* cand = inst + __ldg(top_perm + first);
                if ((__ldg(&cand->mask) & cull) != 0u) {
                    if (sp + 2 > rows) {
                        set_err(err, RQ_DERR_STACK);
                        done = true;
                    } else {
                        const float4* rp = reinterpret_cast<const float4*>(rays + id);
                        const float4 o = __ldg(rp), d = __ldg(rp + 1);
                        const float4* mp = reinterpret_cast<const float4*>(cand->inv);
                        const float4 a = __ldg(mp), b = __ldg(mp + 1), c = __ldg(mp + 2);
                        oo = F3{((a.x * o.x + a.y * o.y) + a.z * o.z) + a.w, ((b.x * o.x + b.y * o.y) + b.z * o.z) + b.w,
                                ((c.x * o.x + c.y * o.y) + c.z * o.z) + c.w};
                        od = F3{(a.x * d.x + a.y * d.y) + a.z * d.z, (b.x * d.x + b.y * d.y) + b.z * d.z,
                                (c.x * d.x + c.y * d.y) + c.z * d.z};
                        sr = slab_setup(oo, od);
                        if (!MT) w = wt_setup(od);
                        nodes = cand->nodes;
                        in = cand;
                        if (top.left) stk[(sp++) * kTT] = top.pack();
                        stk[(sp++) * kTT] = kLeave;
                        top.root();
                    }
                }
            } else {
                const rq_triangle* tris = in->tris;
                const uint32_t cntl = ((uint32_t(pend) >> 27) & 15u) + 1u;
                for (uint32_t p = first; p < first + cntl; ++p) {
                    const float4* tp = reinterpret_cast<const float4*>(tris + p);
                    const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                    const F3 v0{a.x, a.y, a.z}, v1{b.x, b.y, b.z}, v2{c.x, c.y, c.z};
                    float t, u, v;
                    const bool ok =
                        MT ? mt_test(oo, od, v0, v1, v2, 1e-7f, t, u, v) : wt_test(w, oo, v0, v1, v2, t, u, v);
                    if (ok && t >= tmin && t < best) {
                        best = t;
                        hit = true;
                        hit_inst = __ldg(&in->instance_id);
                        hit_prim = __ldg(in->perm + p);
                        if (ANY) {
                            done = true;
                            break;
                        }
                    }
                }
            }
        }
        // ---- report finished rays
        if (active && (done || (sp == 0 && top.left == 0u))) {
            uint4 out = make_uint4(0u, __float_as_uint(-1.0f), 0xffffffffu, 0xffffffffu);
            if (hit) out = make_uint4(1u, __float_as_uint(best), hit_inst, hit_prim);
            reinterpret_cast<uint4*>(hits)[id] = out;
            active = false;
        }
    }
}

}  // namespace

int rq_launch_instance_boxes(rq_ctx* ctx, const TlasInst* inst, const float* fwd, uint32_t n, float* tri9,
                             cudaStream_t st) {
    k_instance_boxes<<<(n + 127) / 128, 128, 0, st>>>(inst, fwd, n, tri9);
    return rq_cuda_status(ctx, cudaGetLastError(), "instance boxes launch");
}

int rq_launch_trace_tlas(rq_ctx* ctx, const rq_tlas* t, const rq_ray* rays, uint32_t n, uint32_t flags,
                         uint32_t cull_mask, rq_hit* hits, cudaStream_t st) {
    if (n == 0) return RQ_OK;
    const bool any = flags & RQ_TRACE_ANY, mt = flags & RQ_TRI_MT;
    const size_t smem = size_t(t->rows) * kTT * (t->wide && !any ? 8 : 4);
    auto k = any       ? (mt ? k_trace_tlas<true, true, false> : k_trace_tlas<true, false, false>)
             : t->wide ? (mt ? k_trace_tlas<false, true, true> : k_trace_tlas<false, false, true>)
                       : (mt ? k_trace_tlas<false, true, false> : k_trace_tlas<false, false, false>);
    cudaError_t e = cudaSuccess;
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTT, smem);
    if (e == cudaSuccess) {
        const uint32_t fill = uint32_t(ctx->num_sms) * uint32_t(per_sm > 0 ? per_sm : 1);
        const uint32_t share = ((n + fill - 1) / fill + 31u) & ~31u;
        const uint32_t per_block = std::max(uint32_t(kTT), std::min(share, kTlasMaxRays));
        k<<<(n + per_block - 1) / per_block, kTT, smem, st>>>(t->top->nodes4, t->top->perm, t->d_inst, rays, n,
                                                               cull_mask, per_block, hits, t->rows, ctx->d_err);
        e = cudaGetLastError();
    }
    return rq_cuda_status(ctx, e, "tlas trace launch");
}
