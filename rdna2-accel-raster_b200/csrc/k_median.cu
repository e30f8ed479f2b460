// k_median.cu — the reference's median-split build (SoftwareBVH::build,
// common/software_bvh.hpp:35-175) on the GPU, for callers that need its tree
// topology (rq_build with RQ_BUILD_MEDIAN).
//
// The reference recurses: a node over primitives [start, end) is a leaf when
// it holds at most max_leaf of them or when its centroids span less than
// 1e-6 on every axis; otherwise the longest centroid axis (ties keep the
// lower axis) is split at mid = (start + end) / 2 by std::nth_element, the
// left child getting the (mid - start) smallest centroids on that axis.
// Nodes are written depth-first, left child at parent + 1.
//
// Splits at mid give children of floor and ceil half the count, so where the
// nodes of a level lie follows from n alone: node j of level L covers the range
// reached by halving [0, n) along the bits of j (med_range), and it exists
// unless a node above it is a leaf.  The primitives are sorted once per axis
// by centroid (one batch of three stable radix sorts of the order-preserving
// key); a node's centroid bounds are then the ends of its three sorted ranges,
// and its left set is the first (mid - start) entries of the range sorted on
// the chosen axis.  A stable partition of the other two orders by that
// membership keeps every node's ranges sorted for the next level.  When no
// centroid value repeats inside a node on its split axis, the left and right
// sets are the ones nth_element produces, so node boxes, child links, leaf
// offsets and counts equal the reference's; the order inside a leaf (left
// unspecified by nth_element) is the x order.
//
//  k_med_setup   centroids, the three sorts' keys
//  k_med_flags   a level's split axes; each primitive's side   } the levels of
//  k_med_part    the partition of the orders                   } ranges > kSub
//  k_med_block   every range of at most kSub primitives in one block: its
//                levels in shared memory, triangles and permutation in their
//                final order, its nodes in pre-order (links relative)
//  k_med_top     boxes, sizes and pre-order positions of the nodes above
//  k_med_out     the blocks' nodes to their places
// What bounds it: latency.  Level by level over the whole mesh down to the
// leaves, nine launches each, the build was 203 launches and 1.49 ms at 99,458
// triangles; now two launches a level above kSub and one below.
// Everything is stream-ordered (no host synchronisation, so the build can be
// captured in a CUDA graph): the host knows the ranges' sizes.
#include <algorithm>

#include "build_core.cuh"
#include "rq_device.cuh"
#include "rq_internal.h"

namespace {

constexpr int kT = 256;
constexpr int kPartItems = 8;
constexpr uint32_t kPartTile = kT * kPartItems;  // positions per block of a global level
constexpr uint32_t kSub = 1024;                  // largest range a block finishes alone
constexpr int kSubT = 512;
constexpr uint32_t kFlagAgg = 1u << 30, kFlagPrefix = 2u << 30, kValueMask = (1u << 30) - 1;
constexpr uint32_t kSpinLimit = 1u << 21;

// A node's state: its split axis, a leaf, or nothing (inside a leaf).
constexpr uint32_t kLeaf = 3u, kNone = 4u;

struct MedScratch {
    uint32_t* keys[2];   // 3 x stride each
    uint32_t* order[2];  // 3 x stride each: the sorts' values, then the levels' orders in turn
    size_t stride;
    float4* cent;        // centroids
    uint8_t* left;       // per primitive: left of its node's split
    uint32_t* local;     // per primitive: its index in its block's range
    float4* rec;         // 4N: two float4 per node, a block's from 4 * start on
    uint32_t* state;     // per node of the levels above the blocks (level L from 2^L - 1 on)
    uint32_t* size;      // the same, and the blocks' level: nodes in the subtree
    uint32_t* pre;       // pre-order position
    float4* box;         // two per node
    uint32_t* words;     // sort scratch
    uint32_t* sync;      // the levels' look-back statuses and tickets (zeroed)
    size_t sync_words;
};

// Number of levels of ranges larger than kSub; level L's largest range.
uint32_t top_levels(uint32_t n) {
    uint32_t t = 0;
    for (uint32_t c = n; c > kSub; c = (c + 1) / 2) ++t;
    return t;
}
uint32_t part_tiles(uint32_t n, uint32_t L) {
    uint32_t c = n;
    for (uint32_t k = 0; k < L; ++k) c = (c + 1) / 2;
    return (c + kPartTile - 1) / kPartTile;
}

size_t carve_med(uintptr_t base, uint32_t n, MedScratch& m) {
    Carve c{base, 0};
    const size_t N = n ? n : 1;
    const uint32_t T = top_levels(uint32_t(N));
    const size_t heap = size_t(2) << T;
    m.stride = (N + 63) & ~size_t(63);
    for (int k = 0; k < 2; ++k) m.keys[k] = c.take<uint32_t>(3 * m.stride);
    for (int k = 0; k < 2; ++k) m.order[k] = c.take<uint32_t>(3 * m.stride);
    m.cent = c.take<float4>(N);
    m.left = c.take<uint8_t>(N);
    m.local = c.take<uint32_t>(N);
    m.rec = c.take<float4>(4 * N);
    m.state = c.take<uint32_t>(heap);
    m.size = c.take<uint32_t>(heap);
    m.pre = c.take<uint32_t>(heap);
    m.box = c.take<float4>(2 * heap);
    m.words = c.take<uint32_t>(rq_sort_words(uint32_t(N), 3));
    m.sync_words = 0;
    for (uint32_t L = 0; L < T; ++L) m.sync_words += (size_t(3) << L) * (part_tiles(uint32_t(N), L) + 1);
    m.sync = c.take<uint32_t>(m.sync_words);
    return c.off + 256;
}

inline uint32_t grid(uint32_t n, int sms) {
    const uint32_t b = (n + kT - 1) / kT;
    return std::max(1u, std::min(b, uint32_t(sms) * 8u));
}

__device__ __forceinline__ float comp(const float4& v, uint32_t a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// Range of node j of level L: [s, s + c).
__device__ __forceinline__ void med_range(uint32_t n, uint32_t L, uint32_t j, uint32_t& s, uint32_t& c) {
    s = 0;
    c = n;
    for (uint32_t b = L; b-- > 0;) {
        const uint32_t h = c / 2;
        if ((j >> b) & 1u) {
            s += h;
            c -= h;
        } else {
            c = h;
        }
    }
}

// The reference's choice for a node's centroid extents: the longest axis (the
// lower one of equals), or a leaf where all are below 1e-6.
__device__ __forceinline__ uint32_t split_axis(float ex, float ey, float ez) {
    uint32_t axis = 0;
    float mx = ex;
    if (ey > mx) {
        axis = 1;
        mx = ey;
    }
    if (ez > mx) {
        axis = 2;
        mx = ez;
    }
    return mx < 1e-6f ? kLeaf : axis;
}

// centroid ((p0+p1)+p2)/3 (software_bvh.hpp:53) and its key on each axis
__global__ void __launch_bounds__(kT) k_med_setup(const float* __restrict__ pos, uint32_t sf,
                                                  const uint32_t* __restrict__ idx, uint32_t n, MedScratch m) {
    for (uint32_t t = blockIdx.x * kT + threadIdx.x; t < n; t += gridDim.x * kT) {
        rq::F3 p0, p1, p2;
        rq::load_tri(pos, sf, idx, t, p0, p1, p2);
        const float4 c = rq::centroid(p0, p1, p2);
        m.cent[t] = c;
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) {
            m.keys[0][a * m.stride + t] = rq::f2o(comp(c, a));
            m.order[0][a * m.stride + t] = t;
        }
    }
}

// Level L, blocks of one node's positions: the node's state, and for a split
// the side of every primitive.  `cur`: the order buffer the level starts from.
__global__ void __launch_bounds__(kT) k_med_flags(uint32_t n, uint32_t L, uint32_t tiles, MedScratch m, int cur) {
    __shared__ uint32_t s_state;
    const uint32_t j = blockIdx.x / tiles, t = blockIdx.x % tiles;
    uint32_t s, c;
    med_range(n, L, j, s, c);
    const uint32_t* ord = cur ? m.order[1] : m.order[0];
    if (threadIdx.x == 0) {
        uint32_t st = kNone;
        if (L == 0 || m.state[(1u << (L - 1)) - 1u + (j >> 1)] < kLeaf) {
            float ext[3];
#pragma unroll
            for (uint32_t a = 0; a < 3; ++a)
                ext[a] = comp(m.cent[ord[a * m.stride + s + c - 1]], a) - comp(m.cent[ord[a * m.stride + s]], a);
            st = split_axis(ext[0], ext[1], ext[2]);
        }
        if (t == 0) m.state[(1u << L) - 1u + j] = st;
        s_state = st;
    }
    __syncthreads();
    if (s_state >= kLeaf) return;
    const uint32_t* o = ord + s_state * m.stride + s;
    const uint32_t h = c / 2, i1 = min((t + 1) * kPartTile, c);
    for (uint32_t i = t * kPartTile + threadIdx.x; i < i1; i += kT) m.left[o[i]] = i < h ? 1 : 0;
}

// Level L: the order of axis blockIdx.y, stably partitioned inside every
// splitting node (copied where the node does not split or this is its axis).
// A node's tiles are taken in order by a ticket and meet by look-back.
__global__ void __launch_bounds__(kT) k_med_part(uint32_t n, uint32_t L, uint32_t tiles, MedScratch m, int cur,
                                                 uint32_t* sync, uint32_t* err) {
    __shared__ uint32_t s_tile, s_prefix, s_warp[kT / 32];
    const uint32_t j = blockIdx.x / tiles, a = blockIdx.y, seg = (a << L) + j;
    uint32_t* ticket = sync + seg;
    uint32_t* status = sync + (3u << L) + size_t(seg) * tiles;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = tiles > 1 ? atomicAdd(ticket, 1u) : 0u;
    __syncthreads();
    const uint32_t t = s_tile;
    uint32_t s, c;
    med_range(n, L, j, s, c);
    const uint32_t* in = (cur ? m.order[1] : m.order[0]) + a * m.stride + s;
    uint32_t* out = (cur ? m.order[0] : m.order[1]) + a * m.stride + s;
    const uint32_t base = t * kPartTile + threadIdx.x * kPartItems;
    uint32_t prim[kPartItems];
    uint32_t bits = 0;
    const uint32_t st = m.state[(1u << L) - 1u + j];
    const bool move = st < kLeaf && st != a;
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) prim[i] = base + i < c ? in[base + i] : 0u;
    if (!move) {
#pragma unroll
        for (int i = 0; i < kPartItems; ++i)
            if (base + i < c) out[base + i] = prim[i];
        return;
    }
#pragma unroll
    for (int i = 0; i < kPartItems; ++i)
        if (base + i < c && m.left[prim[i]]) bits |= 1u << i;
    // the block's exclusive prefix of left counts
    const uint32_t mine = __popc(bits);
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (int(lane) >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t v = lane < kT / 32 ? s_warp[lane] : 0u;
        const uint32_t own = v;
#pragma unroll
        for (int o = 1; o < kT / 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (int(lane) >= o) v += y;
        }
        if (lane < kT / 32) s_warp[lane] = v - own;
        const uint32_t total = __shfl_sync(0xffffffffu, v, kT / 32 - 1);
        uint32_t acc = 0;
        if (t > 0) {
            if (lane == 0) rq::st_release(status + t, kFlagAgg | total);
            uint32_t spins = 0;
            for (int t0 = int(t) - 1;; t0 -= 32) {
                const int p = t0 - int(lane);
                uint32_t w = kFlagPrefix;  // before tile 0
                if (p >= 0)
                    while (!((w = rq::ld_acquire(status + p)) & ~kValueMask))
                        if (++spins > kSpinLimit) {
                            rq::set_err(err, RQ_DERR_SCAN_LOOKBACK);
                            w = kFlagPrefix;
                            break;
                        }
                const uint32_t pm = __ballot_sync(0xffffffffu, (w & ~kValueMask) == kFlagPrefix);
                uint32_t val = w & kValueMask;
                if (pm && int(lane) > __ffs(pm) - 1) val = 0u;
                acc += __reduce_add_sync(0xffffffffu, val);
                if (pm) break;
            }
        }
        if (lane == 0) {
            if (tiles > 1) rq::st_release(status + t, kFlagPrefix | (acc + total));
            s_prefix = acc;
        }
    }
    __syncthreads();
    uint32_t lr = s_prefix + s_warp[warp] + x - mine;
    const uint32_t h = c / 2;
#pragma unroll
    for (int i = 0; i < kPartItems; ++i) {
        if (base + i >= c) break;
        const bool l = (bits >> i) & 1u;
        out[l ? lr : h + (base + i - lr)] = prim[i];
        lr += l;
    }
}

// ------------------------------------------------------------ a block's range
struct SubShared {
    float cen[3][kSub];         // centroids, by local index (position in the x order at the start)
    float box[6][kSub];         // by position: a primitive's box, then its leaf's, then the node's that starts there
    uint32_t gid[kSub];
    uint16_t ord[2][3][kSub];   // local indices
    uint32_t mask[3][kSub / 32];
    uint32_t first[3][kSub / 32];
    uint16_t size[2 * kSub];    // per node (level l from 2^l - 1 on)
    uint16_t pre[2 * kSub];
    uint8_t state[2 * kSub];
    uint8_t left[kSub];
};

__global__ void __launch_bounds__(kSubT, 2) k_med_block(const float* __restrict__ pos, uint32_t sf,
                                                        const uint32_t* __restrict__ idx, uint32_t n, uint32_t T,
                                                        uint32_t max_leaf, MedScratch m, int cur, rq_triangle* tris,
                                                        uint32_t* __restrict__ perm, uint32_t* counts) {
    extern __shared__ __align__(16) char s_raw[];
    SubShared& S = *reinterpret_cast<SubShared*>(s_raw);
    const uint32_t j = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t s0, c0;
    med_range(n, T, j, s0, c0);
    const bool dead = T > 0 && m.state[(1u << (T - 1)) - 1u + (j >> 1)] >= kLeaf;
    // levels below this range's node: the largest range of the last fits a leaf
    uint32_t levels = 0;
    for (uint32_t c = c0; c > max_leaf; c = (c + 1) / 2) ++levels;
    const uint32_t* ord = (cur ? m.order[1] : m.order[0]) + s0;
    for (uint32_t i = threadIdx.x; i < c0; i += kSubT) {
        const uint32_t g = ord[i];
        const float4 ce = m.cent[g];
        S.gid[i] = g;
        S.cen[0][i] = ce.x;
        S.cen[1][i] = ce.y;
        S.cen[2][i] = ce.z;
        S.ord[0][0][i] = uint16_t(i);
        m.local[g] = i;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < c0; i += kSubT) {
        S.ord[0][1][i] = uint16_t(m.local[ord[m.stride + i]]);
        S.ord[0][2][i] = uint16_t(m.local[ord[2 * m.stride + i]]);
    }
    __syncthreads();
    // this thread's positions, and the range of the node each lies in
    constexpr int kPer = kSub / kSubT;
    uint32_t ps[kPer], pc[kPer], pj[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        ps[k] = 0;
        pc[k] = c0;
        pj[k] = 0;
    }
    int buf = 0;
    for (uint32_t l = 0; l <= levels; ++l) {
        const uint32_t heap = (1u << l) - 1u;
        for (uint32_t q = threadIdx.x; q < (1u << l); q += kSubT) {
            uint32_t st = kNone;
            if (l == 0 ? !dead : S.state[((1u << (l - 1)) - 1u) + (q >> 1)] < kLeaf) {
                uint32_t s, c;
                med_range(c0, l, q, s, c);
                st = kLeaf;
                if (c > max_leaf) {
                    float ext[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a)
                        ext[a] = S.cen[a][S.ord[buf][a][s + c - 1]] - S.cen[a][S.ord[buf][a][s]];
                    st = split_axis(ext[0], ext[1], ext[2]);
                }
            }
            S.state[heap + q] = uint8_t(st);
        }
        __syncthreads();
        if (l == levels) break;
        // sides, and each axis's mask of left positions
        uint32_t st[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = k * kSubT + threadIdx.x;
            st[k] = i < c0 ? S.state[heap + pj[k]] : kNone;
            if (st[k] < kLeaf) S.left[S.ord[buf][st[k]][i]] = i < ps[k] + pc[k] / 2;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = k * kSubT + threadIdx.x;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const uint32_t b = __ballot_sync(0xffffffffu, st[k] < kLeaf && S.left[S.ord[buf][a][i]]);
                if (lane == 0) S.mask[a][i >> 5] = b;
            }
        }
        __syncthreads();
        if (warp < 3) {
            const uint32_t own = __popc(S.mask[warp][lane]);
            uint32_t x = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (int(lane) >= o) x += y;
            }
            S.first[warp][lane] = x - own;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = k * kSubT + threadIdx.x;
            if (i >= c0) continue;
            const uint32_t s = ps[k], h = pc[k] / 2;
#pragma unroll
            for (uint32_t a = 0; a < 3; ++a) {
                const uint16_t v = S.ord[buf][a][i];
                uint32_t to = i;
                if (st[k] < kLeaf && st[k] != a) {
                    const uint32_t lr = S.first[a][i >> 5] + __popc(S.mask[a][i >> 5] & ((1u << (i & 31u)) - 1u)) -
                                        S.first[a][s >> 5] - __popc(S.mask[a][s >> 5] & ((1u << (s & 31u)) - 1u));
                    to = (S.mask[a][i >> 5] >> (i & 31u)) & 1u ? s + lr : s + h + (i - s - lr);
                }
                S.ord[buf ^ 1][a][to] = v;
            }
            // the range of the child the position falls in
            if (i < s + h) {
                pc[k] = h;
                pj[k] = 2 * pj[k];
            } else {
                ps[k] = s + h;
                pc[k] -= h;
                pj[k] = 2 * pj[k] + 1;
            }
        }
        buf ^= 1;
        __syncthreads();
    }
    // triangles and permutation in the final order; boxes by position
    for (uint32_t i = threadIdx.x; i < c0; i += kSubT) {
        const uint32_t g = S.gid[S.ord[buf][0][i]];
        rq::F3 p0, p1, p2;
        rq::load_tri(pos, sf, idx, g, p0, p1, p2);
        float4* t = reinterpret_cast<float4*>(tris + s0 + i);
        t[0] = make_float4(p0.x, p0.y, p0.z, 0.0f);
        t[1] = make_float4(p1.x, p1.y, p1.z, 0.0f);
        t[2] = make_float4(p2.x, p2.y, p2.z, 0.0f);
        perm[s0 + i] = g;
        S.box[0][i] = fminf(fminf(p0.x, p1.x), p2.x);
        S.box[1][i] = fminf(fminf(p0.y, p1.y), p2.y);
        S.box[2][i] = fminf(fminf(p0.z, p1.z), p2.z);
        S.box[3][i] = fmaxf(fmaxf(p0.x, p1.x), p2.x);
        S.box[4][i] = fmaxf(fmaxf(p0.y, p1.y), p2.y);
        S.box[5][i] = fmaxf(fmaxf(p0.z, p1.z), p2.z);
    }
    // sizes bottom-up, pre-order positions top-down
    for (uint32_t l = levels + 1; l-- > 0;) {
        const uint32_t heap = (1u << l) - 1u, below = (2u << l) - 1u;
        for (uint32_t q = threadIdx.x; q < (1u << l); q += kSubT) {
            const uint32_t st = S.state[heap + q];
            S.size[heap + q] =
                uint16_t(st == kNone ? 0u : (st == kLeaf ? 1u : 1u + S.size[below + 2 * q] + S.size[below + 2 * q + 1]));
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) S.pre[0] = 0;
    __syncthreads();
    for (uint32_t l = 0; l < levels; ++l) {
        const uint32_t heap = (1u << l) - 1u, below = (2u << l) - 1u;
        for (uint32_t q = threadIdx.x; q < (1u << l); q += kSubT) {
            if (S.state[heap + q] >= kLeaf) continue;
            const uint32_t p = S.pre[heap + q];
            S.pre[below + 2 * q] = uint16_t(p + 1u);
            S.pre[below + 2 * q + 1] = uint16_t(p + 1u + S.size[below + 2 * q]);
        }
        __syncthreads();
    }
    // boxes bottom-up (a node's where its range starts), node records
    float4* rec = m.rec + 4 * size_t(s0);
    uint32_t biggest = 0;
    for (uint32_t l = levels + 1; l-- > 0;) {
        const uint32_t heap = (1u << l) - 1u, below = (2u << l) - 1u;
        for (uint32_t q = threadIdx.x; q < (1u << l); q += kSubT) {
            const uint32_t st = S.state[heap + q];
            if (st == kNone) continue;
            uint32_t s, c;
            med_range(c0, l, q, s, c);
            float b[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) b[k] = S.box[k][s];
            const uint32_t step = st == kLeaf ? 1u : c / 2, end = st == kLeaf ? c : c / 2 + 1u;
            for (uint32_t i = step; i < end; i += step) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    b[k] = fminf(b[k], S.box[k][s + i]);
                    b[k + 3] = fmaxf(b[k + 3], S.box[k + 3][s + i]);
                }
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) S.box[k][s] = b[k];
            const uint32_t p = S.pre[heap + q];
            int32_t lc = int32_t(p + 1u), rc;
            if (st == kLeaf) {
                lc = int32_t(~(s0 + s));
                rc = int32_t(c);
                biggest = max(biggest, c);
            } else {
                rc = int32_t(S.pre[below + 2 * q + 1]);
            }
            rec[2 * p] = make_float4(b[0], b[1], b[2], __int_as_float(lc));
            rec[2 * p + 1] = make_float4(b[3], b[4], b[5], __int_as_float(rc));
        }
        __syncthreads();
    }
    biggest = __reduce_max_sync(0xffffffffu, biggest);
    if (lane == 0 && biggest) atomicMax(counts + 3, biggest);
    // the range's own box and size (a range inside a leaf has no nodes)
    if (dead && warp == 0) {
        float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
        for (uint32_t i = lane; i < c0; i += 32)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                b[k] = fminf(b[k], S.box[k][i]);
                b[k + 3] = fmaxf(b[k + 3], S.box[k + 3][i]);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                b[k] = fminf(b[k], __shfl_xor_sync(0xffffffffu, b[k], o));
                b[k + 3] = fmaxf(b[k + 3], __shfl_xor_sync(0xffffffffu, b[k + 3], o));
            }
        __syncwarp();
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < 6; ++k) S.box[k][0] = b[k];
        __syncwarp();
    }
    if (threadIdx.x == 0) {
        const uint32_t v = (1u << T) - 1u + j;
        m.size[v] = S.size[0];
        m.box[2 * v] = make_float4(S.box[0][0], S.box[1][0], S.box[2][0], 0.0f);
        m.box[2 * v + 1] = make_float4(S.box[3][0], S.box[4][0], S.box[5][0], 0.0f);
    }
}

// The nodes above the blocks, level by level in one block: boxes and sizes up,
// positions down, the nodes themselves.
__global__ void __launch_bounds__(1024) k_med_top(uint32_t n, uint32_t T, MedScratch m, rq_bvh2_node* __restrict__ out,
                                                  uint32_t* counts) {
    for (uint32_t L = T; L-- > 0;) {
        const uint32_t heap = (1u << L) - 1u, below = (2u << L) - 1u;
        for (uint32_t j = threadIdx.x; j < (1u << L); j += 1024) {
            const uint32_t v = heap + j, l = below + 2 * j, r = l + 1, st = m.state[v];
            const float4 la = m.box[2 * l], lb = m.box[2 * l + 1], ra = m.box[2 * r], rb = m.box[2 * r + 1];
            m.box[2 * v] = make_float4(fminf(la.x, ra.x), fminf(la.y, ra.y), fminf(la.z, ra.z), 0.0f);
            m.box[2 * v + 1] = make_float4(fmaxf(lb.x, rb.x), fmaxf(lb.y, rb.y), fmaxf(lb.z, rb.z), 0.0f);
            m.size[v] = st == kNone ? 0u : (st == kLeaf ? 1u : 1u + m.size[l] + m.size[r]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        m.pre[0] = 0;
        counts[0] = m.size[0];
    }
    __syncthreads();
    for (uint32_t L = 0; L < T; ++L) {
        const uint32_t heap = (1u << L) - 1u, below = (2u << L) - 1u;
        for (uint32_t j = threadIdx.x; j < (1u << L); j += 1024) {
            const uint32_t v = heap + j, l = below + 2 * j, r = l + 1, st = m.state[v];
            if (st == kNone) continue;
            const uint32_t p = m.pre[v];
            int32_t lc = int32_t(p + 1u), rc;
            if (st == kLeaf) {
                uint32_t s, c;
                med_range(n, L, j, s, c);
                lc = int32_t(~s);
                rc = int32_t(c);
                atomicMax(counts + 3, c);
            } else {
                m.pre[l] = p + 1u;
                m.pre[r] = p + 1u + m.size[l];
                rc = int32_t(p + 1u + m.size[l]);
            }
            const float4 a = m.box[2 * v], b = m.box[2 * v + 1];
            float4* o = reinterpret_cast<float4*>(out + p);
            o[0] = make_float4(a.x, a.y, a.z, __int_as_float(lc));
            o[1] = make_float4(b.x, b.y, b.z, __int_as_float(rc));
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kT) k_med_out(uint32_t n, uint32_t T, MedScratch m, rq_bvh2_node* __restrict__ out) {
    const uint32_t v = (1u << T) - 1u + blockIdx.x, size = m.size[v];
    if (size == 0) return;
    uint32_t s, c;
    med_range(n, T, blockIdx.x, s, c);
    const float4* rec = m.rec + 4 * size_t(s);
    const uint32_t p0 = m.pre[v];
    float4* o = reinterpret_cast<float4*>(out + p0);
    for (uint32_t k = threadIdx.x; k < size; k += kT) {
        float4 a = rec[2 * k], b = rec[2 * k + 1];
        if (__float_as_int(a.w) >= 0) {  // inner: links relative to the block
            a.w = __int_as_float(__float_as_int(a.w) + int32_t(p0));
            b.w = __int_as_float(__float_as_int(b.w) + int32_t(p0));
        }
        o[2 * k] = a;
        o[2 * k + 1] = b;
    }
}

}  // namespace

int rq_launch_build_median(rq_ctx* ctx, rq_bvh* bvh, const float* pos, uint32_t stride_bytes, const uint32_t* idx,
                           uint32_t n, uint32_t max_leaf, bool collapse, cudaStream_t st) {
    BuildScratch s;
    MedScratch m;
    const size_t bs = rq_build_scratch_carve(nullptr, n, s);
    const size_t need = bs + carve_med(0, n, m);
    int rc = rq_ensure_scratch(ctx, need, st);
    if (rc) return rc;
    rq_build_scratch_carve(ctx->scratch, n, s);
    carve_med(reinterpret_cast<uintptr_t>(ctx->scratch) + ((bs + 255) & ~size_t(255)), n, m);
    const uint32_t sf = stride_bytes / 4;
    cudaError_t e = cudaMemsetAsync(bvh->d_counts, 0, 4 * sizeof(uint32_t), st);
    if (e == cudaSuccess && m.sync_words) e = cudaMemsetAsync(m.sync, 0, sizeof(uint32_t) * m.sync_words, st);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_med_block, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(SubShared)));
    if (e != cudaSuccess) return rq_cuda_status(ctx, e, "median build setup");
    k_med_setup<<<grid(n, ctx->num_sms), kT, 0, st>>>(pos, sf, idx, n, m);
    int cur = 0;
    rc = rq_launch_sort(ctx, SortIO{{m.keys[0], m.keys[1]}, {m.order[0], m.order[1]}, m.stride, m.words}, n, 32, 3, st,
                        &cur);
    if (rc) return rc;
    const uint32_t T = top_levels(n);
    uint32_t* sync = m.sync;
    for (uint32_t L = 0; L < T; ++L) {
        const uint32_t tiles = part_tiles(n, L);
        k_med_flags<<<tiles << L, kT, 0, st>>>(n, L, tiles, m, cur);
        k_med_part<<<dim3(tiles << L, 3), kT, 0, st>>>(n, L, tiles, m, cur, sync, ctx->d_err);
        sync += (size_t(3) << L) * (tiles + 1);
        cur ^= 1;
    }
    k_med_block<<<1u << T, kSubT, sizeof(SubShared), st>>>(pos, sf, idx, n, T, max_leaf, m, cur, bvh->tris, bvh->perm,
                                                           bvh->d_counts);
    k_med_top<<<1, 1024, 0, st>>>(n, T, m, bvh->nodes2, bvh->d_counts);
    k_med_out<<<1u << T, kT, 0, st>>>(n, T, m, bvh->nodes2);
    rc = rq_cuda_status(ctx, cudaGetLastError(), "median build");
    if (rc) return rc;
    if (collapse) return rq_launch_collapse(ctx, bvh, s, st);
    return RQ_OK;
}
