// trace_engine.cuh — persistent traversal with per-lane ray refill.
//
// Every lane of a warp owns one ray at a time.  Ray ids come from a global
// counter in chunks (one atomic per chunk); whenever enough lanes are idle,
// a ballot and a rank within the idle mask hand them the next ids, so a warp
// keeps its rays in flight until the ids run out.  Each round:
//   1. node phase — lanes without a parked leaf take the next child of the
//      deepest open node: an inner child is opened (its four boxes tested, the
//      hit ones noted with their order), a leaf is parked; the phase ends when
//      no lane searches, or few do while others wait with leaves;
//   2. leaf phase — lanes test their parked leaf's triangles in order;
//   3. lanes that have nothing left to visit, or whose any-hit ray found a
//      hit, report the result to the ray source and become idle.
// Per ray the children are visited in exactly the order of a sequential
// depth-first traversal (closest hit: nearest child first, ties by slot; any
// hit: by slot), so results do not depend on which lane or round a ray runs
// in and match the oracle's traversal bit for bit.
//
// The open nodes of a ray are a path, so the stack holds one entry per open
// node with children left — its index and their order — rather than one per
// child: depth + 1 rows where 3 * depth + 1 were needed (15 for 43 on the
// 2.5M-triangle frame's tree; the shared memory goes to the L1).  Where a
// child leads (child_index, child_count) is read when its turn comes, not for
// all four when the node is opened: the box test needs six of the node's
// eight rows, an unvisited child costs nothing, and an any-hit node's entry
// is its hit mask as it stands.  Measured against an entry per child with its
// target resolved when its node is opened: 2^20 incoherent rays on 999,698
// triangles (closest hit) 511 -> 412 us; the 1080p frame's 27.1M shadow and AO
// rays 6.17 -> 5.59 ms; 2.07M camera rays on 8.3M triangles 1.94 -> 1.64 ms.
// What bounds it now is the L1 (LSU wavefronts at 72 % of their peak on the
// shadow rays, 83 % on the incoherent ones: lanes of a warp read different
// nodes) together with instruction issue (69 % and 52 %).
// Tried here and no faster: 32-byte loads of two rows with the planes picked
// by selects (shadow 5.75 ms, incoherent 393 us), packed two-wide plane
// distances (spills), 56 or 48 registers for 36 or 40 warps per SM (shadow
// 5.73 / 5.76 ms), speculative traversal, refilling inside the node loop,
// staging the top levels in shared memory.
//
// A ray source provides:
//   uint32_t total;                                 number of ray ids
//   bool make(uint32_t id, Ray& r, Meta& m);        false = no ray for this id
//   void finish(uint32_t id, const Meta& m, const Ray& r, const Hit& h);
//   optional: kRoundEnd = true and void round_end(bool finished, const Meta& m).
#pragma once

#include <type_traits>

#include "rq_device.cuh"
#include "rq_internal.h"

namespace rq {

constexpr int32_t kNoLeaf = 0;  // a parked leaf always has bit 31 set
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kChunk = 32;  // default ray ids per refill atomic

struct Ray {
    F3 o, d;
    float tmin, tmax;
    // set by sources that trace many BVHs in one launch (Src::kMulti)
    const rq_bvh4_node* nodes;
    const rq_triangle* tris;
    bool any;  // per-ray any hit (ANY == kAnyPerRay)
};

// ANY template argument: 0 closest hit, 1 any hit, kAnyPerRay = Ray::any.
constexpr int kAnyPerRay = 2;

template <class Src, class = void>
struct IsMulti {
    static constexpr bool value = false;
};
template <class Src>
struct IsMulti<Src, decltype(void(Src::kMulti))> {
    static constexpr bool value = Src::kMulti;
};

// Sources with kRoundEnd get round_end(finished, meta) once per round from
// all 32 lanes together (finished: this lane reported a ray this round;
// meta: that ray's), e.g. to count completions with one atomic per group.
template <class Src, class = void>
struct HasRoundEnd {
    static constexpr bool value = false;
};
template <class Src>
struct HasRoundEnd<Src, decltype(void(Src::kRoundEnd))> {
    static constexpr bool value = Src::kRoundEnd;
};

struct Hit {
    bool hit;
    float t;
    uint32_t idx;  // leaf-order primitive index
    float u, v;
    uint32_t boxes, tris;
};

// ---------------------------------------------------------------- open nodes
// The deepest open node of a ray: its index (kRootRef: the root itself is the
// next child) and the children left to visit.  MASK (any-hit kernels): `left`
// is a mask of slots, visited from the lowest.  Otherwise a sequence of 3-bit
// fields 4 | slot, the next one lowest; at most four, and at most three once
// the first has been taken, which is when the node can go to the stack.
// Stack entries are node << 4 | mask or node << 9 | sequence in 32 bits: the
// sequence form holds node indices below 2^23 (RQ_NARROW_NODES), so trees with
// more room than that run with 64-bit entries (WIDE).
constexpr int32_t kRootRef = -1;

template <bool MASK, bool WIDE>
struct OpenNode {
    using Entry = typename std::conditional<WIDE, unsigned long long, uint32_t>::type;
    static constexpr int kBits = MASK ? 4 : 9;
    int32_t node;
    uint32_t left;

    __device__ __forceinline__ void root() {
        node = kRootRef;
        left = 4u;  // (one child, whichever the form)
    }
    __device__ __forceinline__ Entry pack() const { return (Entry(uint32_t(node)) << kBits) | left; }
    __device__ __forceinline__ void unpack(Entry e) {
        node = int32_t(e >> kBits);
        left = uint32_t(e) & ((1u << kBits) - 1u);
    }
    __device__ __forceinline__ uint32_t take() {
        if (MASK) {
            const uint32_t k = uint32_t(__ffs(left)) - 1u;
            left &= left - 1u;
            return k;
        }
        const uint32_t k = left & 3u;
        left >>= 3;
        return k;
    }
};

// The order of a node's hit children as a sequence: near to far with ties by
// slot (sorted), or by slot.  A hit child may lie at infinity (a ray without
// an end, a plane distance past the float range), so distance alone does not
// keep a missed child behind the hit ones.  Its hit bit is tested where it
// could come first; with MIXED rays (sorted or not, by ray) it stands in there
// as NaN, which took serving's mix 4,956 us for 4,983, and a million scattered
// closest-hit rays 414 for 412.
template <bool MIXED>
__host__ __device__ __forceinline__ uint32_t child_sequence(uint32_t hitm, const float (&tk)[4], bool sorted) {
    float first[4], second[4];
    bool hit[4];
    for (int k = 0; k < 4; ++k) {
        hit[k] = (hitm >> k) & 1u;
        const float t = sorted ? tk[k] : 0.0f;
        second[k] = hit[k] ? t : INFINITY;
        first[k] = MIXED ? (hit[k] ? t : NAN) : second[k];
    }
    // child i is hit and comes before child j
    auto before = [&](int i, int j) { return uint32_t((MIXED || hit[i]) && first[i] <= second[j]); };
    const uint32_t p01 = before(0, 1), p02 = before(0, 2), p03 = before(0, 3), p12 = before(1, 2), p13 = before(1, 3),
                   p23 = before(2, 3);
    const uint32_t r[4] = {3u - (p01 + p02 + p03), p01 + 2u - (p12 + p13), p02 + p12 + 1u - p23, p03 + p13 + p23};
    uint32_t s = 0;
    for (uint32_t k = 0; k < 4; ++k) s |= hit[k] ? (4u | k) << (3u * r[k]) : 0u;
    return s;
}

// Where child `slot` of `node` leads: child_index, child_count.
__device__ __forceinline__ void child_of(const rq_bvh4_node* __restrict__ nodes, int32_t node, uint32_t slot,
                                         int32_t& ci, int32_t& cc) {
    ci = 0;
    cc = -1;  // (the root)
    if (node >= 0) {
        const int32_t* q = reinterpret_cast<const int32_t*>(nodes + node) + 24 + slot;
        ci = __ldg(q);
        cc = __ldg(q + 4);
    }
}

// Leaves of the node phase: it ends once at most kFewSearch lanes search while
// kLeafWait hold a leaf (measured on B200: 8 and 8; without it the 1080p
// frame's shadow pass was 3 %, the depth-AO pass 13 % slower, 16 and 8 were
// 3 % and 4 % slower than 8 and 8).  few: kFewSearch, or 0 where the whole phase
// is short.
constexpr int kFewSearch = 8, kLeafWait = 8;

// Stack rows for trees of `depth` 4-wide levels, as the host knows them, whose
// handle may be rebuilt in place before the host reads the new depth: d levels
// leave at most d - 1 open nodes behind.  Four levels to spare, and otherwise
// what the stack of children before held (3 * (depth + 2) + 1 entries) up to 24
// rows, trees of 25 levels: a 2,000-triangle mesh 7 levels deep that contracts
// toward a point is rebuilt to 20.  Up to 24 rows cost nothing, since the
// shared memory they need comes in steps: camera rays on 8.3M triangles 2,245
// us with 18 rows, 2,247 with 24, 2,266 with 28 and 2,306 with 46.
inline int rebuild_rows(uint32_t depth) {
    return int(depth + 4u > 24u ? depth + 4u : (3u * depth + 7u < 24u ? 3u * depth + 7u : 24u));
}

// A parked leaf holds RQ_MAX_LEAF primitives.  The host refuses trees with
// larger leaves by its copy of the counts; after an in-place rebuild that it
// has not read back the live count (counts[3]) tells.  One thread of a launch.
__device__ __forceinline__ void check_leaves(const uint32_t* __restrict__ counts, uint32_t* err) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && __ldg(counts + 3) > RQ_MAX_LEAF) set_err(err, RQ_DERR_LEAF);
}

// stk: this lane's column of `rows` stack entries, STRIDE apart.  CHUNK: ray
// ids taken per atomic.  refill_min: idle lanes get new rays only once at
// least this many lanes of the warp are idle (or all are), so that lanes join
// in groups and a warp's rays stay closer in position and direction.  lanes:
// lanes of a warp that take rays, as many ids at a time (32: all, CHUNK ids).
template <int ANY, bool MT, bool STATS, int STRIDE, class Src, int CHUNK = int(kChunk), bool WIDE = false>
__device__ __forceinline__ void trace_persistent(const rq_bvh4_node* __restrict__ nodes,
                                                 const rq_triangle* __restrict__ tris, Src& src, uint32_t* ctr,
                                                 typename OpenNode<ANY == 1, WIDE>::Entry* stk, int rows,
                                                 uint32_t* err, int refill_min = 1, uint32_t lanes = 32u,
                                                 int few = kFewSearch) {
    const uint32_t takers = lanes == 32u ? kFull : (1u << lanes) - 1u;
    const uint32_t chunk = lanes == 32u ? uint32_t(CHUNK) : lanes;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    // warp-uniform chunk of ray ids
    uint32_t next = 0, end = 0;
    bool exhausted = false;
    // lane state
    bool active = false;
    uint32_t rid = 0;
    typename Src::Meta meta;
    Ray ray;
    SlabRay sr;
    WtRay w;
    float best = 0.0f;
    OpenNode<ANY == 1, WIDE> top;  // the deepest open node
    top.left = 0;
    int sp = 0;  // entries on the stack
    Hit h;
    h.hit = false;
    h.t = 0.0f;
    h.idx = kNoHit;
    h.u = h.v = 0.0f;
    h.boxes = h.tris = 0;

    for (;;) {
        // ---- new rays for idle lanes, once refill_min of them are idle
        uint32_t idle = __ballot_sync(kFull, !active) & takers;
        const bool go = __popc(idle) >= refill_min || idle == takers;
        while (go && idle && !exhausted) {
            if (next == end) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(ctr, chunk);
                base = __shfl_sync(kFull, base, 0);
                if (base >= src.total) {
                    exhausted = true;
                    break;
                }
                next = base;
                end = min(base + chunk, src.total);
            }
            const uint32_t take = min(uint32_t(__popc(idle)), end - next);
            const uint32_t rank = __popc(idle & lt_mask);
            const bool mine = ((idle >> lane) & 1u) && rank < take;
            if (mine) {
                rid = next + rank;
                if (src.make(rid, ray, meta)) {
                    active = true;
                    sr.ix = safe_inv(ray.d.x);
                    sr.iy = safe_inv(ray.d.y);
                    sr.iz = safe_inv(ray.d.z);
                    sr.ox = ray.o.x * sr.ix;
                    sr.oy = ray.o.y * sr.iy;
                    sr.oz = ray.o.z * sr.iz;
                    if (!MT) w = wt_setup(ray.d);
                    best = ray.tmax;
                    h.hit = false;
                    h.idx = kNoHit;
                    h.u = h.v = 0.0f;
                    h.boxes = h.tris = 0;
                    top.root();
                    sp = 0;
                }
            }
            next += take;
            // lanes whose id made no ray (a light behind the surface, an
            // empty pixel) take the next id at once
            idle = __ballot_sync(kFull, !active) & takers;
        }
        if (!__any_sync(kFull, active)) {
            if (exhausted) break;
            continue;
        }

        // ---- node phase
        int32_t leaf = kNoLeaf;
        for (;;) {
            const bool search = active && leaf == kNoLeaf && (top.left != 0u || sp > 0);
            const uint32_t sm = __ballot_sync(kFull, search);
            if (!sm) break;
            if (__popc(sm) <= few && __popc(__ballot_sync(kFull, leaf != kNoLeaf)) >= kLeafWait) break;
            if (!search) continue;
            if (top.left == 0u) top.unpack(stk[(--sp) * STRIDE]);
            const uint32_t slot = top.take();
            const rq_bvh4_node* nb = IsMulti<Src>::value ? ray.nodes : nodes;
            int32_t ci, cc;
            child_of(nb, top.node, slot, ci, cc);
            if (cc >= 0) {  // a leaf (or an empty slot whose point box the ray met)
                if (cc > 0) leaf = int32_t(0x80000000u | (uint32_t(cc - 1) << 27) | uint32_t(~ci));
                continue;
            }
            float tk[4];
            const uint32_t hitm = box4_hits<false>(GlobalRows{reinterpret_cast<const float4*>(nb + ci)}, sr, ray.tmin,
                                                   best, tk);
            if (STATS) h.boxes += 4;
            if (hitm) {
                if (top.left) {
                    if (sp < rows)
                        stk[(sp++) * STRIDE] = top.pack();
                    else
                        set_err(err, RQ_DERR_STACK);  // deeper than the host knew
                }
                top.node = ci;
                top.left = ANY == 1 ? hitm : child_sequence<ANY == kAnyPerRay>(hitm, tk, ANY == 0 || !ray.any);
            }
        }

        // ---- leaf phase
        bool done = false;
        if (active && leaf != kNoLeaf) {
            const uint32_t first = uint32_t(leaf) & 0x07ffffffu;
            const uint32_t cntl = ((uint32_t(leaf) >> 27) & 15u) + 1u;
            for (uint32_t p = first; p < first + cntl; ++p) {
                const float4* tp = reinterpret_cast<const float4*>((IsMulti<Src>::value ? ray.tris : tris) + p);
                const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                const F3 v0{a.x, a.y, a.z}, v1{b.x, b.y, b.z}, v2{c.x, c.y, c.z};
                if (STATS) ++h.tris;
                float t, u, v;
                const bool ok = MT ? mt_test(ray.o, ray.d, v0, v1, v2, 1e-7f, t, u, v)
                                   : wt_test(w, ray.o, v0, v1, v2, t, u, v);
                if (ok && t >= ray.tmin && t < best) {
                    best = t;
                    h.hit = true;
                    h.idx = p;
                    h.u = u;
                    h.v = v;
                    if (ANY == 1 || (ANY == kAnyPerRay && ray.any)) {
                        done = true;
                        break;
                    }
                }
            }
        }

        // ---- report finished rays
        bool fin = false;
        if (active && (done || (sp == 0 && top.left == 0u))) {
            h.t = best;
            src.finish(rid, meta, ray, h);
            active = false;
            fin = true;
        }
        if constexpr (HasRoundEnd<Src>::value) {
            __syncwarp();
            src.round_end(fin, meta);
        }
    }
}

}  // namespace rq
