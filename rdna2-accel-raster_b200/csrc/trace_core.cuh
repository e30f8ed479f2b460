// trace_core.cuh — the engine's 4-wide traversal of one ray by one thread
// from start to end (the schedule for one coherent closest-hit ray per thread,
// such as camera rays; trace_engine.cuh is the schedule that refills lanes).
// Its open nodes, their entries and the visit order are trace_engine.cuh's, so
// results are identical.  Each thread's stack lives in shared memory with a
// stride of the block size, so the entries of one warp fall in distinct banks.
#pragma once

#include "trace_engine.cuh"

namespace rq {

struct TraceResult {
    float t;        // nearest accepted distance (tmax when nothing was hit)
    uint32_t idx;   // leaf-order primitive index, kNoHit for a miss
    float u, v;     // barycentrics of v1 and v2
};

// stk: this thread's column of `rows` stack entries, STRIDE apart.
template <bool MT, int STRIDE, bool WIDE>
__device__ __forceinline__ void trace_ray(const rq_bvh4_node* __restrict__ nodes,
                                          const rq_triangle* __restrict__ tris,
                                          typename OpenNode<false, WIDE>::Entry* stk, int rows, F3 o, F3 d, float tmin,
                                          float tmax, TraceResult& res, uint32_t* err) {
    SlabRay sr;
    sr.ix = safe_inv(d.x);
    sr.iy = safe_inv(d.y);
    sr.iz = safe_inv(d.z);
    sr.ox = o.x * sr.ix;
    sr.oy = o.y * sr.iy;
    sr.oz = o.z * sr.iz;
    WtRay w;
    if (!MT) w = wt_setup(d);
    float best = tmax;
    res.idx = kNoHit;
    res.u = res.v = 0.0f;
    OpenNode<false, WIDE> top;
    top.root();
    int sp = 0;
    while (top.left != 0u || sp > 0) {
        if (top.left == 0u) top.unpack(stk[(--sp) * STRIDE]);
        const uint32_t slot = top.take();
        int32_t ci, cc;
        child_of(nodes, top.node, slot, ci, cc);
        if (cc < 0) {
            float tk[4];
            const uint32_t hitm = box4_hits<true>(GlobalRows{reinterpret_cast<const float4*>(nodes + ci)}, sr, tmin,
                                                  best, tk);
            if (hitm) {
                if (top.left) {
                    if (sp < rows)
                        stk[(sp++) * STRIDE] = top.pack();
                    else
                        set_err(err, RQ_DERR_STACK);  // deeper than the host knew
                }
                top.node = ci;
                top.left = child_sequence<false>(hitm, tk, true);
            }
        } else {  // a leaf (or an empty slot whose point box the ray met)
            const uint32_t first = uint32_t(~ci);
            for (uint32_t p = first; p < first + uint32_t(cc); ++p) {
                const float4* tp = reinterpret_cast<const float4*>(tris + p);
                const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                const F3 v0{a.x, a.y, a.z}, v1{b.x, b.y, b.z}, v2{c.x, c.y, c.z};
                float t, u, v;
                const bool ok = MT ? mt_test(o, d, v0, v1, v2, 1e-7f, t, u, v) : wt_test_fixed(w, o, v0, v1, v2, t, u, v);
                if (ok && t >= tmin && t < best) {
                    best = t;
                    res.idx = p;
                    res.u = u;
                    res.v = v;
                }
            }
        }
    }
    res.t = best;
}

}  // namespace rq
