// k_small.cu — the whole LBVH build of a small mesh in one block.
//
// Up to kSmallMax triangles the build of k_build.cu is a chain of 14 launches
// whose steps are short: each waits for the last one's tail, and every
// dependent load goes to L2 (the 4-wide collapse alone took 47 us at 4,096
// triangles, five dependent loads per node and level).  Here one block of
// 1,024 threads takes the mesh through the same steps with everything but the
// vertices and the outputs in shared memory: centroids and Morton codes, a
// stable radix sort, the radix tree, the pre-order positions, the boxes (of the
// emitted nodes only, at their pre-order places), the 4-wide collapse.
// The rules are those of build_core.cuh, so the bytes equal k_build.cu's.
// 4,096 triangles 143 -> 75 us, 256 triangles 88 -> 28 us (the sort 15 and 8 us
// of them, the vertex gathers 14 us, the collapse 10 us).  Above 4,096 the
// shared memory is full, and one SM gathering the vertices would be the bound.
// Trees of more than kNodes binary nodes (possible above kNodes / 2 triangles)
// keep their node arrays in the context's scratch instead.
#include <atomic>

#include "build_core.cuh"
#include "rq_device.cuh"
#include "rq_internal.h"

namespace {

using namespace rq;

constexpr int kT = 1024, kWarps = kT / 32;
constexpr uint32_t kSmallMax = 4096;  // primitives
constexpr uint32_t kItems = kSmallMax / kT;
constexpr uint32_t kNodes = 4096;     // binary nodes in shared memory
constexpr uint32_t kLevels = 120;     // 4-wide levels (as the grid-wide collapse)
constexpr uint32_t kNone16 = 0xffffu;

// Arrays of the emitted tree, by pre-order position.
struct TreeArrays {
    float* box;      // 6 planes of `cap`: min xyz, max xyz
    float* area;
    uint16_t* link;  // inner: the right child; leaf: the first primitive
    uint16_t* par;
    uint8_t* leaf;   // 0: inner; else the leaf's count
    uint32_t cap;
    // 4-wide nodes, by queue entry (at most cap / 2)
    uint16_t* cand;   // 4 each
    uint16_t* child;  // 4 each: queue entry of an inner candidate
    uint16_t* q;      // binary node
    uint16_t* size;
    uint16_t* pre;
};

struct Shared {
    // the emitted tree, or before it the sort's second buffers and counters
    union {
        struct {
            float box[6][kNodes];
        } t;
        struct {
            uint32_t keys[kSmallMax];
            uint16_t ids[kSmallMax];
            uint16_t cnt[kWarps][256];
        } s;
    } a;
    // the radix tree by split, then the 4-wide nodes
    union {
        struct {
            uint16_t kr[kSmallMax], klo[kSmallMax], khi[kSmallMax];                 // bit 15 of kr: a leaf
            uint16_t par_in[kSmallMax], par_lf[kSmallMax];                          // (parent << 1) | is_right
        } k;
        struct {
            uint16_t cand[4 * kNodes / 2], child[4 * kNodes / 2], q[kNodes / 2], size[kNodes / 2], pre[kNodes / 2];
        } c;
    } b;
    // sorted keys, then the nodes' surface areas
    union {
        uint32_t keys[kSmallMax];
        float area[kNodes];
    } k;
    uint16_t ids[kSmallMax];
    uint16_t c[kSmallMax], A[kSmallMax];  // emission counts and their exclusive scan
    uint16_t link[kNodes], par[kNodes];
    uint8_t leaf[kNodes];
    uint32_t seen[2 * kSmallMax / 32];  // arrivals of the refit
    uint32_t warp[kWarps];
    uint32_t part[4][256];
    uint8_t adj[kSmallMax];  // common prefix of a sorted key and the next
    float red[6][kWarps];
    uint32_t lvl[kLevels + 2];
    uint32_t tail;
};
static_assert(sizeof(Shared) <= 227 * 1024, "one block's shared memory");

// Exclusive scan of one value per thread; *total = the sum.
__device__ __forceinline__ uint32_t scan1024(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (int(lane) >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (int(lane) >= o) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t r = (warp ? s_warp[warp - 1] : 0u) + x - v;
    *total = s_warp[kWarps - 1];
    __syncthreads();
    return r;
}

// Common prefix of sorted keys i and i + 1, by index where they are equal.
__device__ __forceinline__ int delta(const uint32_t* k, uint32_t i) {
    const uint32_t x = k[i] ^ k[i + 1];
    return x ? __clz(x) : 32 + __clz(i ^ (i + 1));
}

// Left-child links above the node whose parent link is `par`.
__device__ __forceinline__ uint32_t left_links(const Shared& S, uint32_t par) {
    uint32_t L = 0;
    while (par != kNone16 && (par & 1u) == 0u) {
        ++L;
        par = S.b.k.par_in[par >> 1];
    }
    return L;
}

struct SmallArgs {
    const float* pos;
    uint32_t sf;
    const uint32_t* idx;
    uint32_t n, max_leaf;
    bool collapse;
    rq_triangle* tris;
    uint32_t* perm;
    uint32_t* skeys;
    rq_bvh2_node* nodes2;
    rq_bvh4_node* nodes4;
    int32_t* map4;
    uint32_t* counts;
    TreeArrays far;  // the node arrays of a tree that does not fit
    uint32_t* err;
};

// f(position, triangle, vertices) for this thread's sorted positions, two
// triangles' loads in flight together.
template <class F>
__device__ __forceinline__ void each_triangle(const SmallArgs& A, const Shared& S, F f) {
#pragma unroll
    for (uint32_t r = 0; r < kItems; r += 2) {
        const uint32_t k0 = r * kT + threadIdx.x, k1 = k0 + kT;
        if (k0 >= A.n) break;
        const uint32_t i0 = S.ids[k0], i1 = k1 < A.n ? S.ids[k1] : i0;
        F3 a0, b0, c0, a1, b1, c1;
        load_tri(A.pos, A.sf, A.idx, i0, a0, b0, c0);
        load_tri(A.pos, A.sf, A.idx, i1, a1, b1, c1);
        f(k0, i0, a0, b0, c0);
        if (k1 < A.n) f(k1, i1, a1, b1, c1);
    }
}

__global__ void __launch_bounds__(kT, 1) k_build_small(const __grid_constant__ SmallArgs A) {
    extern __shared__ __align__(16) char s_raw[];
    Shared& S = *reinterpret_cast<Shared*>(s_raw);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n = A.n;

    // ---- centroids, their bounds, Morton codes
    float4 cen[kItems];
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
        const uint32_t t = r * kT + threadIdx.x;
        if (t >= n) continue;
        F3 p0, p1, p2;
        load_tri(A.pos, A.sf, A.idx, t, p0, p1, p2);
        cen[r] = centroid(p0, p1, p2);
        mn[0] = fminf(mn[0], cen[r].x);
        mn[1] = fminf(mn[1], cen[r].y);
        mn[2] = fminf(mn[2], cen[r].z);
        mx[0] = fmaxf(mx[0], cen[r].x);
        mx[1] = fmaxf(mx[1], cen[r].y);
        mx[2] = fmaxf(mx[2], cen[r].z);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
        if (lane == 0) {
            S.red[k][warp] = mn[k];
            S.red[3 + k][warp] = mx[k];
        }
    }
    for (uint32_t i = threadIdx.x; i < 2 * kSmallMax / 32; i += kT) S.seen[i] = 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = S.red[k][lane];
        mx[k] = S.red[3 + k][lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    }
    {
        const float scale = morton_scale(mn[0], mn[1], mn[2], mx[0], mx[1], mx[2]);
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t t = r * kT + threadIdx.x;
            if (t >= n) continue;
            S.k.keys[t] = morton30(cen[r], mn[0], mn[1], mn[2], scale);
            S.ids[t] = uint16_t(t);
        }
    }

    // ---- stable sort of (code, id): 4 passes of 8 bits.  Warp w holds the
    // positions [128 w, 128 w + 128); buffer 0 is S.k.keys / S.ids.
    for (int pass = 0; pass < 4; ++pass) {
        uint32_t* kin = pass & 1 ? S.a.s.keys : S.k.keys;
        uint16_t* vin = pass & 1 ? S.a.s.ids : S.ids;
        uint32_t* kout = pass & 1 ? S.k.keys : S.a.s.keys;
        uint16_t* vout = pass & 1 ? S.ids : S.a.s.ids;
        const uint32_t shift = 8u * pass;
        for (uint32_t i = threadIdx.x; i < kWarps * 256u / 2u; i += kT) reinterpret_cast<uint32_t*>(S.a.s.cnt)[i] = 0u;
        __syncthreads();
        uint32_t key[kItems], rank[kItems];
        uint16_t val[kItems];
        uint16_t* cnt = S.a.s.cnt[warp];
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t i = warp * (32 * kItems) + r * 32 + lane;
            const bool valid = i < n;
            const uint32_t act = __ballot_sync(0xffffffffu, valid);
            key[r] = rank[r] = 0;
            val[r] = 0;
            if (valid) {
                key[r] = kin[i];
                val[r] = vin[i];
                const uint32_t d = (key[r] >> shift) & 255u;
                uint32_t peers = act;
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const bool bit = (d >> b) & 1u;
                    const uint32_t m = __ballot_sync(act, bit);
                    peers &= bit ? m : ~m;
                }
                const uint32_t below = __popc(peers & ((1u << lane) - 1u)), c = cnt[d];
                __syncwarp(act);
                if (below == 0) cnt[d] = uint16_t(c + __popc(peers));
                rank[r] = c + below;
            }
            __syncwarp();
        }
        __syncthreads();
        // digit d's counts: 4 threads of 8 warps each, then the digits' bases
        const uint32_t d = threadIdx.x & 255u, quarter = threadIdx.x >> 8;
        uint32_t c8[8], own = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            c8[w] = S.a.s.cnt[quarter * 8 + w][d];
            own += c8[w];
        }
        S.part[quarter][d] = own;
        __syncthreads();
        uint32_t run = 0, tot = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t v = S.part[q][d];
            if (q < quarter) run += v;
            tot += v;
        }
        {
            // (every 8 warps hold the 256 digits in order)
            uint32_t x = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (int(lane) >= o) x += y;
            }
            if (lane == 31) S.warp[warp] = x;
            __syncthreads();
            run += x - tot;
            for (uint32_t w = warp & ~7u; w < warp; ++w) run += S.warp[w];
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            S.a.s.cnt[quarter * 8 + w][d] = uint16_t(run);
            run += c8[w];
        }
        __syncthreads();
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t i = warp * (32 * kItems) + r * 32 + lane;
            if (i < n) {
                const uint32_t at = cnt[(key[r] >> shift) & 255u] + rank[r];
                kout[at] = key[r];
                vout[at] = val[r];
            }
        }
        __syncthreads();
    }
    const uint32_t* keys = S.k.keys;

    // ---- the binary radix tree of the sorted codes (Karras's; built from the
    // leaves up as Apetrei 2014: a range's parent splits it off at whichever
    // end shares the longer prefix with its neighbour).  A node is named by
    // its split: the last primitive of its left child.
    for (uint32_t i = threadIdx.x; i < n; i += kT) S.adj[i] = i + 1 < n ? uint8_t(delta(keys, i) + 1) : uint8_t(0);
    __syncthreads();
    // (a thread takes neighbours: all but its last climb end early)
    for (uint32_t k = threadIdx.x * kItems; k < min(n, (threadIdx.x + 1) * kItems); ++k) {
        uint32_t lo = k, hi = k, ref = 0x8000u | k;
        for (;;) {
            const uint32_t dl = lo ? S.adj[lo - 1] : 0u, dr = S.adj[hi];
            uint16_t* mine = ref & 0x8000u ? S.b.k.par_lf + (ref & 0x7fffu) : S.b.k.par_in + ref;
            if (!(dl | dr)) {  // the root
                *mine = kNone16;
                break;
            }
            const bool left = dr > dl;
            const uint32_t p = left ? hi : lo - 1u;
            *mine = uint16_t((p << 1) | (left ? 0u : 1u));
            if (left) {
                S.b.k.klo[p] = uint16_t(lo);
            } else {
                S.b.k.kr[p] = uint16_t(ref);
                S.b.k.khi[p] = uint16_t(hi);
            }
            __threadfence_block();  // this range before the arrival
            if (!((atomicOr(&S.seen[p >> 5], 1u << (p & 31u)) >> (p & 31u)) & 1u)) break;
            __threadfence_block();
            lo = S.b.k.klo[p];
            hi = S.b.k.khi[p];
            ref = p;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 2 * kSmallMax / 32; i += kT) S.seen[i] = 0u;

    // ---- emission counts: the nodes whose range starts at a position, down the left links
    uint32_t sum = 0;
    uint32_t cw[kItems];
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
        const uint32_t k = threadIdx.x * kItems + r;
        cw[r] = 0;
        if (k >= n) continue;
        uint32_t par = S.b.k.par_lf[k], ulo = k;
        while (par != kNone16) {
            const uint32_t p = par >> 1;
            if (uint32_t(S.b.k.khi[p]) - S.b.k.klo[p] + 1u > A.max_leaf) break;
            ulo = S.b.k.klo[p];
            par = S.b.k.par_in[p];
        }
        if (ulo == k) cw[r] = 1u + left_links(S, par);
        S.c[k] = uint16_t(cw[r]);
        sum += cw[r];
    }
    uint32_t total;
    {
        uint32_t run = scan1024(sum, S.warp, &total);
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t k = threadIdx.x * kItems + r;
            if (k < n) S.A[k] = uint16_t(run);
            run += cw[r];
        }
    }
    __syncthreads();

    // ---- the emitted tree's links, by pre-order position
    const bool near = total <= kNodes;
    TreeArrays T = A.far;
    if (near) {
        T.box = &S.a.t.box[0][0];
        T.area = S.k.area;
        T.link = S.link;
        T.par = S.par;
        T.leaf = S.leaf;
        T.cap = kNodes;
    }
    if (threadIdx.x == 0) T.par[0] = kNone16;
    for (uint32_t p = threadIdx.x; p < n; p += kT) {
        if (p + 1 < n && uint32_t(S.b.k.khi[p]) - S.b.k.klo[p] + 1u > A.max_leaf) {
            const uint32_t pre = S.A[S.b.k.klo[p]] + left_links(S, S.b.k.par_in[p]);
            const uint32_t r = S.b.k.kr[p], rpre = S.A[r & 0x8000u ? r & 0x7fffu : uint32_t(S.b.k.klo[r])];
            T.link[pre] = uint16_t(rpre);
            T.leaf[pre] = 0;
            T.par[pre + 1] = uint16_t(pre);
            T.par[rpre] = uint16_t(pre);
        }
        const uint32_t c = S.c[p];
        if (c) {
            uint32_t par = S.b.k.par_lf[p], count = 1;
            while (par != kNone16) {
                const uint32_t cnt = uint32_t(S.b.k.khi[par >> 1]) - S.b.k.klo[par >> 1] + 1u;
                if (cnt > A.max_leaf) break;
                count = cnt;
                par = S.b.k.par_in[par >> 1];
            }
            const uint32_t pre = S.A[p] + c - 1u;
            T.link[pre] = uint16_t(p);
            T.leaf[pre] = uint8_t(count);
        }
    }
    __syncthreads();

    // ---- the leaf order's outputs; boxes: the primitives' by position, then
    // each leaf's at its node (one SM gathers 4,096 triangles' vertices in 9 us,
    // so they are read once here and once for the centroids)
    auto box = [&](int k, uint32_t v) -> float& { return T.box[k * T.cap + v]; };
    each_triangle(A, S, [&](uint32_t k, uint32_t id, F3 a, F3 b, F3 c) {
        float4* tp = reinterpret_cast<float4*>(A.tris + k);
        tp[0] = make_float4(a.x, a.y, a.z, 0.0f);
        tp[1] = make_float4(b.x, b.y, b.z, 0.0f);
        tp[2] = make_float4(c.x, c.y, c.z, 0.0f);
        A.perm[k] = id;
        A.skeys[k] = keys[k];
        box(0, k) = fminf(a.x, fminf(b.x, c.x));
        box(1, k) = fminf(a.y, fminf(b.y, c.y));
        box(2, k) = fminf(a.z, fminf(b.z, c.z));
        box(3, k) = fmaxf(a.x, fmaxf(b.x, c.x));
        box(4, k) = fmaxf(a.y, fmaxf(b.y, c.y));
        box(5, k) = fmaxf(a.z, fmaxf(b.z, c.z));
    });
    __syncthreads();
    {
        float lf[kItems][6];
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t p = r * kT + threadIdx.x;
            if (p >= n || !S.c[p]) continue;
            const uint32_t last = p + T.leaf[S.A[p] + S.c[p] - 1u];
#pragma unroll
            for (int k = 0; k < 6; ++k) lf[r][k] = box(k, p);
            for (uint32_t q = p + 1; q < last; ++q)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    lf[r][k] = fminf(lf[r][k], box(k, q));
                    lf[r][3 + k] = fmaxf(lf[r][3 + k], box(3 + k, q));
                }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t r = 0; r < kItems; ++r) {
            const uint32_t p = r * kT + threadIdx.x;
            if (p >= n || !S.c[p]) continue;
#pragma unroll
            for (int k = 0; k < 6; ++k) box(k, S.A[p] + S.c[p] - 1u) = lf[r][k];
        }
    }
    __syncthreads();
    // ---- and upward: the second child to arrive goes on
    for (uint32_t p = threadIdx.x * kItems; p < min(n, (threadIdx.x + 1) * kItems); ++p) {
        if (!S.c[p]) continue;
        uint32_t v = S.A[p] + S.c[p] - 1u;
        for (;;) {
            const uint32_t up = T.par[v];
            if (up == kNone16) break;
            __threadfence_block();  // v's box before the arrival
            if (!((atomicOr(&S.seen[up >> 5], 1u << (up & 31u)) >> (up & 31u)) & 1u)) break;
            __threadfence_block();
            const uint32_t l = up + 1u, r = T.link[up];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                box(k, up) = fminf(box(k, l), box(k, r));
                box(3 + k, up) = fmaxf(box(3 + k, l), box(3 + k, r));
            }
            v = up;
        }
    }
    __syncthreads();

    // ---- the binary nodes, and their areas (greedy_candidates)
    for (uint32_t v = threadIdx.x; v < total; v += kT) {
        const float b0 = box(0, v), b1 = box(1, v), b2 = box(2, v), b3 = box(3, v), b4 = box(4, v), b5 = box(5, v);
        const uint32_t count = T.leaf[v], link = T.link[v];
        float4* o = reinterpret_cast<float4*>(A.nodes2 + v);
        o[0] = make_float4(b0, b1, b2, __int_as_float(count ? ~int32_t(link) : int32_t(v + 1u)));
        o[1] = make_float4(b3, b4, b5, __int_as_float(count ? int32_t(count) : int32_t(link)));
        const float dx = b3 - b0, dy = b4 - b1, dz = b5 - b2;
        T.area[v] = 2.0f * ((dx * dy + dy * dz) + dz * dx);
    }
    if (threadIdx.x == 0) {
        A.counts[0] = total;
        A.counts[3] = A.max_leaf;
    }
    if (!A.collapse) return;
    __syncthreads();

    // ---- 4-wide nodes, level by level: candidates, inner ones queued
    if (near) {
        T.cand = S.b.c.cand;
        T.child = S.b.c.child;
        T.q = S.b.c.q;
        T.size = S.b.c.size;
        T.pre = S.b.c.pre;
    }
    if (threadIdx.x == 0) {
        T.q[0] = 0;
        S.tail = 1;
        S.lvl[0] = 0;
    }
    __syncthreads();
    uint32_t depth = 0, start = 0, end = 1;
    while (start < end) {
        for (uint32_t e = start + threadIdx.x; e < end; e += kT) {
            const uint32_t u = T.q[e];
            uint32_t c[4] = {u, kNone16, kNone16, kNone16};
            int nc = 1;
            if (!T.leaf[u]) {  // (the root alone can be a leaf)
                c[0] = u + 1u;
                c[1] = T.link[u];
                nc = 2;
            }
#pragma unroll
            for (int it = 0; it < 2; ++it) {
                int best = -1;
                float best_sa = -1.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < nc && !T.leaf[c[i]]) {
                        const float sa = T.area[c[i]];
                        if (sa > best_sa) {
                            best_sa = sa;
                            best = i;
                        }
                    }
                if (best < 0) break;
                uint32_t o = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i == best) o = c[i];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i == best) c[i] = o + 1u;
                    if (i == nc) c[i] = T.link[o];
                }
                ++nc;
            }
            uint32_t inner = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < nc && !T.leaf[c[i]]) inner |= 1u << i;
            uint32_t at = inner ? atomicAdd(&S.tail, uint32_t(__popc(inner))) : 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                T.cand[4 * e + i] = uint16_t(i < nc ? c[i] : kNone16);
                uint32_t ch = kNone16;
                if ((inner >> i) & 1u) {
                    ch = at++;
                    T.q[ch] = uint16_t(c[i]);
                }
                T.child[4 * e + i] = uint16_t(ch);
            }
        }
        __syncthreads();
        ++depth;
        start = end;
        end = S.tail;
        if (threadIdx.x == 0 && depth <= kLevels) S.lvl[depth] = start;
        if (depth >= kLevels && start < end) {
            if (threadIdx.x == 0) set_err(A.err, RQ_DERR_QUEUE);
            return;
        }
        __syncthreads();
    }
    // sizes bottom-up, positions and nodes top-down
    for (uint32_t lv = depth; lv-- > 0;) {
        for (uint32_t e = S.lvl[lv] + threadIdx.x; e < S.lvl[lv + 1]; e += kT) {
            uint32_t s = 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = T.child[4 * e + i];
                if (ch != kNone16) s += T.size[ch];
            }
            T.size[e] = uint16_t(s);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        T.pre[0] = 0;
        A.counts[1] = end;
        A.counts[2] = depth;
    }
    __syncthreads();
    for (uint32_t lv = 0; lv < depth; ++lv) {
        for (uint32_t e = S.lvl[lv] + threadIdx.x; e < S.lvl[lv + 1]; e += kT) {
            uint32_t off = T.pre[e] + 1u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = T.child[4 * e + i];
                if (ch == kNone16) continue;
                T.pre[ch] = uint16_t(off);
                off += T.size[ch];
            }
        }
        __syncthreads();
    }
    for (uint32_t e = threadIdx.x; e < end; e += kT) {
        const uint32_t p = T.pre[e];
        float b[6][4];
        int32_t ci[4], cc[4], m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t c = T.cand[4 * e + i], ch = T.child[4 * e + i];
            ci[i] = cc[i] = 0;
            m[i] = -1;
#pragma unroll
            for (int k = 0; k < 6; ++k) b[k][i] = 0.0f;
            if (c == kNone16) continue;
            m[i] = int32_t(c);
#pragma unroll
            for (int k = 0; k < 6; ++k) b[k][i] = box(k, c);
            if (ch != kNone16) {
                ci[i] = T.pre[ch];
                cc[i] = -1;
            } else {
                ci[i] = ~int32_t(T.link[c]);
                cc[i] = T.leaf[c];
            }
        }
        float4* o = reinterpret_cast<float4*>(A.nodes4 + p);
        o[0] = make_float4(b[0][0], b[0][1], b[0][2], b[0][3]);
        o[1] = make_float4(b[3][0], b[3][1], b[3][2], b[3][3]);
        o[2] = make_float4(b[1][0], b[1][1], b[1][2], b[1][3]);
        o[3] = make_float4(b[4][0], b[4][1], b[4][2], b[4][3]);
        o[4] = make_float4(b[2][0], b[2][1], b[2][2], b[2][3]);
        o[5] = make_float4(b[5][0], b[5][1], b[5][2], b[5][3]);
        reinterpret_cast<int4*>(o)[6] = make_int4(ci[0], ci[1], ci[2], ci[3]);
        reinterpret_cast<int4*>(o)[7] = make_int4(cc[0], cc[1], cc[2], cc[3]);
        reinterpret_cast<int4*>(A.map4)[p] = make_int4(m[0], m[1], m[2], m[3]);
    }
}

}  // namespace

bool rq_small_build(uint32_t n) { return n <= kSmallMax; }

int rq_launch_build_small(rq_ctx* ctx, rq_bvh* bvh, const float* pos, uint32_t stride_bytes, const uint32_t* idx,
                          uint32_t n, uint32_t max_leaf, bool collapse, cudaStream_t st) {
    // node arrays of a tree of more than kNodes nodes (at most 2 * kSmallMax)
    constexpr uint32_t kFar = 2 * kSmallMax;
    SmallArgs a;
    Carve c{0, 0};
    for (int pass = 0; pass < 2; ++pass) {
        a.far.box = c.take<float>(6 * kFar);
        a.far.area = c.take<float>(kFar);
        a.far.link = c.take<uint16_t>(kFar);
        a.far.par = c.take<uint16_t>(kFar);
        a.far.leaf = c.take<uint8_t>(kFar);
        a.far.cap = kFar;
        a.far.cand = c.take<uint16_t>(4 * kFar / 2);
        a.far.child = c.take<uint16_t>(4 * kFar / 2);
        a.far.q = c.take<uint16_t>(kFar / 2);
        a.far.size = c.take<uint16_t>(kFar / 2);
        a.far.pre = c.take<uint16_t>(kFar / 2);
        if (pass) break;
        int rc = rq_ensure_scratch(ctx, c.off + 256, st);
        if (rc) return rc;
        c = Carve{reinterpret_cast<uintptr_t>(ctx->scratch), 0};
    }
    a.pos = pos;
    a.sf = stride_bytes / 4;
    a.idx = idx;
    a.n = n;
    a.max_leaf = max_leaf;
    a.collapse = collapse;
    a.tris = bvh->tris;
    a.perm = bvh->perm;
    a.skeys = bvh->skeys;
    a.nodes2 = bvh->nodes2;
    a.nodes4 = bvh->nodes4;
    a.map4 = bvh->map4;
    a.counts = bvh->d_counts;
    a.err = ctx->d_err;
    // the shared-memory attribute holds for the device once set
    static std::atomic<bool> s_set[64];
    const int dev = ctx->device;
    cudaError_t e = cudaSuccess;
    if (dev < 0 || dev >= 64 || !s_set[dev].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(k_build_small, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(Shared)));
        if (e == cudaSuccess && dev >= 0 && dev < 64) s_set[dev].store(true, std::memory_order_relaxed);
    }
    if (e == cudaSuccess) {
        k_build_small<<<1, kT, sizeof(Shared), st>>>(a);
        e = cudaGetLastError();
    }
    return rq_cuda_status(ctx, e, "small build launch");
}
