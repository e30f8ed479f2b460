// build_core.cuh — the per-element steps of the LBVH build, shared by the
// kernels of k_build.cu / k_collapse.cu (one mesh per launch sequence) and of
// k_forest.cu (all meshes of a batch per launch).  Both call these functions,
// so a mesh built either way has the same bytes.
//
// Loads of data written earlier in the same launch use plain (coherent)
// loads; only the caller's vertex and index buffers go through __ldg.
#pragma once

#include "rq_device.cuh"
#include "rq_internal.h"

namespace rq {

constexpr uint32_t kNoParent = 0xffffffffu;

__device__ __forceinline__ void load_tri(const float* __restrict__ pos, uint32_t sf, const uint32_t* __restrict__ idx,
                                         uint32_t t, F3& p0, F3& p1, F3& p2) {
    uint32_t i0, i1, i2;
    if (idx) {
        i0 = __ldg(idx + 3ull * t);
        i1 = __ldg(idx + 3ull * t + 1);
        i2 = __ldg(idx + 3ull * t + 2);
    } else {
        i0 = 3 * t;
        i1 = 3 * t + 1;
        i2 = 3 * t + 2;
    }
    const float* a = pos + size_t(i0) * sf;
    const float* b = pos + size_t(i1) * sf;
    const float* c = pos + size_t(i2) * sf;
    p0 = {__ldg(a), __ldg(a + 1), __ldg(a + 2)};
    p1 = {__ldg(b), __ldg(b + 1), __ldg(b + 2)};
    p2 = {__ldg(c), __ldg(c + 1), __ldg(c + 2)};
}

// Centroid exactly as SoftwareBVH::build (common/software_bvh.hpp:53).
__device__ __forceinline__ float4 centroid(F3 p0, F3 p1, F3 p2) {
    return make_float4(((p0.x + p1.x) + p2.x) / 3.0f, ((p0.y + p1.y) + p2.y) / 3.0f, ((p0.z + p1.z) + p2.z) / 3.0f,
                       0.0f);
}

// Scale of the Morton grid: 1024 cells over the largest centroid extent.
__device__ __forceinline__ float morton_scale(float lx, float ly, float lz, float hx, float hy, float hz) {
    const float ext = fmaxf(fmaxf(hx - lx, hy - ly), hz - lz);
    return ext > 1e-30f ? 1024.0f / ext : 0.0f;
}

__device__ __forceinline__ uint32_t morton30(float4 c, float lx, float ly, float lz, float scale) {
    return expand10(quantize10(c.x, lx, scale)) * 4u + expand10(quantize10(c.y, ly, scale)) * 2u +
           expand10(quantize10(c.z, lz, scale));
}

__device__ __forceinline__ int kdelta(const uint32_t* k, int n, int i, int j) {
    if (j < 0 || j > n - 1) return -1;
    const uint32_t x = k[i] ^ k[j];
    if (x) return __clz(x);
    return 32 + __clz(uint32_t(i) ^ uint32_t(j));
}

// Karras 2012, internal node i of n sorted keys: children (bit 31 = leaf),
// range, and the parent links of both children ((parent << 1) | is_right).
__device__ __forceinline__ void karras_node(const uint32_t* keys, int n, int i, int32_t* kl, int32_t* kr,
                                            uint32_t* klo, uint32_t* khi, uint32_t* par_in, uint32_t* par_lf) {
    const int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = kdelta(keys, n, i, i - d);
    int lmax = 2;
    while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = kdelta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const bool lleaf = lo == gamma, rleaf = hi == gamma + 1;
    kl[i] = lleaf ? int32_t(0x80000000u | uint32_t(gamma)) : gamma;
    kr[i] = rleaf ? int32_t(0x80000000u | uint32_t(gamma + 1)) : gamma + 1;
    klo[i] = uint32_t(lo);
    khi[i] = uint32_t(hi);
    const uint32_t pl = uint32_t(i) << 1, pr = (uint32_t(i) << 1) | 1u;
    if (lleaf)
        par_lf[gamma] = pl;
    else
        par_in[gamma] = pl;
    if (rleaf)
        par_lf[gamma + 1] = pr;
    else
        par_in[gamma + 1] = pr;
    if (i == 0) par_in[0] = kNoParent;
}

__device__ __forceinline__ uint32_t count_in(const uint32_t* klo, const uint32_t* khi, uint32_t i) {
    return khi[i] - klo[i] + 1u;
}

// Atomic bottom-up refit from the parent link `par` of a node whose box is
// final: at each node the second child to arrive computes the union box and
// continues upward.  The arrival count is an acquire-release add: it publishes
// the box this thread wrote last and, for the second arrival, makes the
// sibling's box visible.
__device__ __forceinline__ void refit_walk_up(uint32_t par, const int32_t* kl, const int32_t* kr,
                                              const uint32_t* par_in, float4* box_in, const float4* box_lf,
                                              uint32_t* refit_flag, uint32_t* err) {
    uint32_t guard = 0;
    while (par != kNoParent) {
        const uint32_t p = par >> 1;
        if (atom_add_acq_rel(&refit_flag[p], 1u) == 0u) break;
        const int32_t a = kl[p], b = kr[p];
        const float4* ba = a < 0 ? box_lf + 2 * size_t(uint32_t(a) & 0x7fffffffu) : box_in + 2 * size_t(a);
        const float4* bb = b < 0 ? box_lf + 2 * size_t(uint32_t(b) & 0x7fffffffu) : box_in + 2 * size_t(b);
        const float4 alo = ld_cg4(ba), ahi = ld_cg4(ba + 1);
        const float4 blo = ld_cg4(bb), bhi = ld_cg4(bb + 1);
        __stcg(box_in + 2 * size_t(p), make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), 0.0f));
        __stcg(box_in + 2 * size_t(p) + 1,
               make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.0f));
        par = par_in[p];
        if (++guard > 128u) {
            set_err(err, RQ_DERR_REFIT);
            break;
        }
    }
}

// ------------------------------------------------- the LBVH's tree, bottom up
// The binary radix tree of the sorted codes (Karras 2012, ties by position)
// built from the leaves up as Apetrei 2014: a range's parent splits it off at
// whichever end shares the longer prefix with its neighbour, so a node needs
// only its own range and the two gaps at its ends, and its box, its place in
// the depth-first order and its children's emission come from the same climb.
// A node is named by its gap: the first position of its right child.
//
// What the climb leaves for the emission, all by position:
//   ch[x]     bits 0..7: emitted nodes whose range starts at x and that are
//             not below another starting there, counted down the left links
//             (c: the inner ones and the emitted leaf; 0: no emitted node);
//             bits 8..15: emitted nodes on the left links of the node with gap
//             x, itself included (h; 0: not emitted)
//   rec[2x]   the node with gap x, if emitted: (min, range start), (max, -)
//   leaf[2x]  the emitted leaf that starts at x: (min, count), (max, -)
// With A the exclusive scan of c, the chain of emitted nodes starting at x
// takes the places A[x] .. A[x] + c[x] - 1, outermost first: the node with gap
// x and range start lo goes to A[lo + 1] - 1 - h, its right child to A[x].
// (Depths stay below 30 + 27 levels, so c and h fit a byte.)
//
// A block takes kTreeLeaves sorted leaves and climbs in shared memory; nodes
// whose sibling lies outside go on in tree_climb_top with the same steps over
// global memory.  The form this replaces searched each node's range (Karras),
// wrote children, ranges and parents to memory, and read them again in the
// refit and in two chains of dependent loads per leaf and node.  On 8.3M
// triangles (1,132 us before, 593 us now, scan included): search 235 us, leaves
// and refit 549 -> 382, its top 113 -> 62, node writes 165 -> 111; 512 meshes of
// 4.73M triangles together 733 -> 383.  The climb's blocks are bound by the L1
// (LSU wavefronts at 73 %: scattered vertex reads 40 % of the time, shared
// memory the rest); 512 leaves per block doubled the top's time, 128 threads of
// 8 leaves took 493 us.
constexpr uint32_t kTreeT = 256, kTreeItems = 4, kTreeLeaves = kTreeT * kTreeItems;
constexpr uint32_t kTreeBlocks = 5;  // per SM (registers and shared memory; 4: 422 us for 382 us on 8.3M)

struct TreeOut {
    rq_triangle* tris;
    uint32_t *perm, *keys;
    uint16_t* ch;
    float4 *rec, *leaf;
    // unfinished nodes: (min, other end), (max, h) at the end that touches the
    // sibling, and one arrival bit per gap (zeroed)
    float4* slot;
    uint32_t* seen;
};

// Slots are padded so that a warp's neighbouring quadruples fall in distinct banks.
__device__ __forceinline__ uint32_t tree_slot(uint32_t i) { return i + (i >> 5); }

struct TreeShared {
    float box[6][kTreeLeaves + kTreeLeaves / 32];
    uint8_t adj[kTreeLeaves + 1];   // common prefix + 1 across the gap before a position; 0: none
    uint32_t seen[kTreeLeaves / 16 + 1];  // arrivals per gap: bit 0 the left child, bit 1 the right one
    uint32_t count, base;
    union {
        float4 stage[kTreeT / 32][96];  // a warp's 32 triangles as they are written; then
        struct {
            uint16_t end[kTreeLeaves];  // an unfinished node's other end
            uint8_t h[kTreeLeaves];
            uint16_t ch[kTreeLeaves + 2];
            uint16_t list[kTreeLeaves + 2];  // (gap << 1) | is_right
        };
    };
};

// Common prefix + 1 of the sorted codes on both sides of the gap before x (0: no gap).
__device__ __forceinline__ uint32_t tree_gap(const uint32_t* keys, uint32_t n, uint32_t x) {
    if (x == 0u || x >= n) return 0u;
    const uint32_t d = keys[x - 1u] ^ keys[x];
    return d ? uint32_t(__clz(d)) + 1u : 33u + uint32_t(__clz((x - 1u) ^ x));
}

struct TreeBox {
    float v[6];  // min, max
};
__device__ __forceinline__ TreeBox tree_union(const TreeBox& a, const TreeBox& b) {
    TreeBox r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.v[k] = fminf(a.v[k], b.v[k]);
        r.v[3 + k] = fmaxf(a.v[3 + k], b.v[3 + k]);
    }
    return r;
}
__device__ __forceinline__ void tree_put(float4* at, const TreeBox& b, uint32_t lo_w, uint32_t hi_w) {
    __stcg(at, make_float4(b.v[0], b.v[1], b.v[2], __uint_as_float(lo_w)));
    __stcg(at + 1, make_float4(b.v[3], b.v[4], b.v[5], __uint_as_float(hi_w)));
}

// A finished node [lo, hi] with gap x: its records and its children's.
// Returns the word ch[x] gets; h: in, the left child's; out, the node's.
__device__ __forceinline__ uint32_t tree_emit(const TreeOut& O, uint32_t max_leaf, uint32_t lo, uint32_t x, uint32_t hi,
                                              const TreeBox& l, const TreeBox& r, const TreeBox& b, uint32_t& h,
                                              uint32_t hr) {
    if (hi - lo + 1u <= max_leaf) {
        h = 0u;
        return 0u;
    }
    h += 1u;
    tree_put(O.rec + 2 * size_t(x), b, lo, 0u);
    if (x - lo <= max_leaf) tree_put(O.leaf + 2 * size_t(lo), l, x - lo, 0u);
    if (hi - x + 1u <= max_leaf) tree_put(O.leaf + 2 * size_t(x), r, hi - x + 1u, 0u);
    return (h << 8) | (hr + 1u);
}
// The root's own place (and the leaf it is, if it is one).
__device__ __forceinline__ uint32_t tree_root(const TreeOut& O, uint32_t max_leaf, uint32_t n, const TreeBox& b,
                                              uint32_t h) {
    if (n <= max_leaf) tree_put(O.leaf, b, n, 0u);
    return h + 1u;
}

// The vertices of the warp's 32 triangles (lane's triangle: id), component by
// component: neighbouring lanes read neighbouring words, 11 rows per load
// instead of 32.  stage[3 * lane + c] = vertex c of the lane's triangle (its
// fourth word holds the vertex index).
__device__ __forceinline__ void tree_gather(float4* stage, uint32_t id, const float* __restrict__ pos, uint32_t sf,
                                            const uint32_t* __restrict__ idx) {
    const uint32_t lane = threadIdx.x & 31u;
    float* s = reinterpret_cast<float*>(stage);
#pragma unroll
    for (uint32_t j = 0; j < 3; ++j) {
        const uint32_t e = j * 32u + lane, t = e / 3u, i = __shfl_sync(0xffffffffu, id, int(t)) * 3u + (e - 3u * t);
        s[4u * e + 3u] = __uint_as_float(idx ? __ldg(idx + i) : i);
    }
    __syncwarp();
    float v[9];
#pragma unroll
    for (uint32_t j = 0; j < 9; ++j) {
        const uint32_t f = j * 32u + lane, e = f / 3u;
        v[j] = __ldg(pos + size_t(__float_as_uint(s[4u * e + 3u])) * sf + (f - 3u * e));
    }
#pragma unroll
    for (uint32_t j = 0; j < 9; ++j) {
        const uint32_t f = j * 32u + lane, e = f / 3u;
        s[4u * e + (f - 3u * e)] = v[j];
    }
    __syncwarp();
}

// The leaves [L0, min(L0 + kTreeLeaves, n)) by one block of kTreeT threads:
// the leaf-ordered triangles, permutation and keys, and every node whose range
// lies inside.  On return S.list[0 .. S.count) holds the unfinished nodes
// (gaps from L0), their slots written to O.slot.
__device__ __forceinline__ void tree_climb_block(TreeShared& S, uint32_t L0, uint32_t n, const float* __restrict__ pos,
                                                 uint32_t sf, const uint32_t* __restrict__ idx, uint32_t max_leaf,
                                                 const uint32_t* __restrict__ keys, const uint32_t* __restrict__ ids,
                                                 const TreeOut& O) {
    const uint32_t m = min(kTreeLeaves, n - L0), lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kTreeLeaves / 16 + 1; i += kTreeT) S.seen[i] = 0u;
    for (uint32_t i = threadIdx.x; i <= m; i += kTreeT) S.adj[i] = uint8_t(tree_gap(keys, n, L0 + i));
    if (threadIdx.x == 0) S.count = 0u;
    float4* stage = S.stage[warp];
#pragma unroll 1
    for (uint32_t r = 0; r < kTreeItems; ++r) {
        const uint32_t i0 = (r * (kTreeT / 32) + warp) * 32u, i = i0 + lane;
        if (i0 >= m) break;
        const uint32_t id = ids[L0 + min(i, m - 1u)];
        tree_gather(stage, id, pos, sf, idx);
        const float4 a = stage[3 * lane], b = stage[3 * lane + 1], c = stage[3 * lane + 2];
        if (i < m) {
            O.perm[L0 + i] = id;
            O.keys[L0 + i] = keys[L0 + i];
            const uint32_t s = tree_slot(i);
            S.box[0][s] = fminf(a.x, fminf(b.x, c.x));
            S.box[1][s] = fminf(a.y, fminf(b.y, c.y));
            S.box[2][s] = fminf(a.z, fminf(b.z, c.z));
            S.box[3][s] = fmaxf(a.x, fmaxf(b.x, c.x));
            S.box[4][s] = fmaxf(a.y, fmaxf(b.y, c.y));
            S.box[5][s] = fmaxf(a.z, fmaxf(b.z, c.z));
        }
        float4* out = reinterpret_cast<float4*>(O.tris + L0 + i0);
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
            const uint32_t e = j * 32u + lane;
            float4 v = stage[e];
            v.w = 0.0f;
            if (i0 + e / 3u < m) out[e] = v;
        }
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= m; i += kTreeT) S.ch[i] = 0;
    __syncthreads();

    // ---- the climb: a thread takes four neighbours, all but its last climb end early
    auto load = [&](uint32_t at) {
        TreeBox b;
        const uint32_t s = tree_slot(at);
#pragma unroll
        for (int k = 0; k < 6; ++k) b.v[k] = S.box[k][s];
        return b;
    };
#pragma unroll 1
    for (uint32_t j = 0; j < kTreeItems; ++j) {
        const uint32_t k = threadIdx.x * kTreeItems + j;
        if (k >= m) break;
        uint32_t lo = k, hi = k, h = 0;  // positions from L0
        TreeBox b = load(k);
        for (;;) {
            const uint32_t dl = S.adj[lo], dr = S.adj[hi + 1u];
            if (!(dl | dr)) {
                S.ch[0] = uint16_t(tree_root(O, max_leaf, n, b, h));
                break;
            }
            const bool right = dl > dr;
            const uint32_t x = right ? lo : hi + 1u;
            volatile uint32_t* sw = S.seen + (x >> 4);
            const uint32_t sh = 2u * (x & 15u), own = (right ? 2u : 1u) << sh, other = (right ? 1u : 2u) << sh;
            if (*sw & other) {
                atomicOr(const_cast<uint32_t*>(sw), own);
            } else {
                const uint32_t at = right ? lo : hi, s = tree_slot(at);
#pragma unroll
                for (int q = 0; q < 6; ++q) S.box[q][s] = b.v[q];
                S.end[at] = uint16_t(right ? hi : lo);
                S.h[at] = uint8_t(h);
                __threadfence_block();  // the node before its arrival
                if (!(atomicOr(const_cast<uint32_t*>(sw), own) & other)) break;
            }
            __threadfence_block();
            const uint32_t at = right ? x - 1u : x, he = S.h[at];
            const TreeBox sib = load(at);
            uint32_t hr = he;
            if (right) {
                lo = S.end[at];
                hr = h;
                h = he;
            } else {
                hi = S.end[at];
            }
            const TreeBox l = right ? sib : b, r = right ? b : sib;
            b = tree_union(l, r);
            S.ch[x] = uint16_t(tree_emit(O, max_leaf, L0 + lo, L0 + x, L0 + hi, l, r, b, h, hr));
        }
    }
    __syncthreads();

    // ---- the emission words; the nodes whose sibling has not come
    for (uint32_t i = threadIdx.x; i <= m; i += kTreeT) {
        if (i < m) O.ch[L0 + i] = S.ch[i];
        const uint32_t a = (S.seen[i >> 4] >> (2u * (i & 15u))) & 3u;
        if (a == 1u || a == 2u) {
            const uint32_t at = a == 1u ? i - 1u : i;
            S.list[atomicAdd(&S.count, 1u)] = uint16_t((i << 1) | (a - 1u));
            tree_put(O.slot + 2 * size_t(L0 + at), load(at), L0 + S.end[at], S.h[at]);
        }
    }
    __syncthreads();
}

// Carries an unfinished node on over global memory (entry: (gap << 1) | is_right).
__device__ __forceinline__ void tree_climb_top(uint32_t entry, uint32_t n, uint32_t max_leaf,
                                               const uint32_t* __restrict__ keys, const TreeOut& O) {
    auto load = [&](uint32_t at, TreeBox& b, uint32_t& end, uint32_t& h) {
        const float4 lo = ld_cg4(O.slot + 2 * size_t(at)), hi = ld_cg4(O.slot + 2 * size_t(at) + 1);
        b = TreeBox{{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z}};
        end = __float_as_uint(lo.w);
        h = __float_as_uint(hi.w);
    };
    uint32_t x = entry >> 1;
    bool right = entry & 1u;
    TreeBox b;
    uint32_t lo = x, hi = x - 1u, h;
    if (right)
        load(x, b, hi, h);
    else
        load(x - 1u, b, lo, h);
    for (;;) {
        const uint32_t bit = 1u << (x & 31u);
        if (!(atom_or_acq_rel(O.seen + (x >> 5), bit) & bit)) return;
        TreeBox sib;
        uint32_t end, he, hr;
        load(right ? x - 1u : x, sib, end, he);
        if (right) {
            lo = end;
            hr = h;
            h = he;
        } else {
            hi = end;
            hr = he;
        }
        const TreeBox l = right ? sib : b, r = right ? b : sib;
        b = tree_union(l, r);
        O.ch[x] = uint16_t(tree_emit(O, max_leaf, lo, x, hi, l, r, b, h, hr));
        const uint32_t dl = tree_gap(keys, n, lo), dr = tree_gap(keys, n, hi + 1u);
        if (!(dl | dr)) {
            O.ch[0] = uint16_t(tree_root(O, max_leaf, n, b, h));
            return;
        }
        right = dl > dr;
        x = right ? lo : hi + 1u;
        tree_put(O.slot + 2 * size_t(right ? lo : hi), b, right ? hi : lo, h);
    }
}

// The nodes that position x emits: the inner node with gap x and the leaf that
// starts at x.  Returns the number of nodes emitted up to x.
template <class Scan>
__device__ __forceinline__ uint32_t tree_write(uint32_t x, const TreeOut& O, const Scan& A, rq_bvh2_node* out) {
    const uint32_t w = O.ch[x], c = w & 255u, h = w >> 8, a = A[x];
    if (h) {
        const float4 lo = ldg4(O.rec + 2 * size_t(x)), hi = ldg4(O.rec + 2 * size_t(x) + 1);
        const uint32_t at = A[__float_as_uint(lo.w) + 1u] - 1u - h;
        float4* o = reinterpret_cast<float4*>(out + at);
        o[0] = make_float4(lo.x, lo.y, lo.z, __int_as_float(int32_t(at + 1u)));
        o[1] = make_float4(hi.x, hi.y, hi.z, __int_as_float(int32_t(a)));
    }
    if (c) {
        const float4 lo = ldg4(O.leaf + 2 * size_t(x)), hi = ldg4(O.leaf + 2 * size_t(x) + 1);
        float4* o = reinterpret_cast<float4*>(out + a + c - 1u);
        o[0] = make_float4(lo.x, lo.y, lo.z, __int_as_float(~int32_t(x)));
        o[1] = make_float4(hi.x, hi.y, hi.z, lo.w);  // (count)
    }
    return a + c;
}

// ------------------------------------------------------------- collapse
struct N2 {
    float mn[3], mx[3];
    int32_t l, r;
};

__device__ __forceinline__ N2 load_n2(const rq_bvh2_node* n2, int32_t i) {
    const float4* p = reinterpret_cast<const float4*>(n2 + i);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    N2 o;
    o.mn[0] = a.x;
    o.mn[1] = a.y;
    o.mn[2] = a.z;
    o.l = __float_as_int(a.w);
    o.mx[0] = b.x;
    o.mx[1] = b.y;
    o.mx[2] = b.z;
    o.r = __float_as_int(b.w);
    return o;
}

// The collapse's surface area of a node.
__device__ __forceinline__ float node_area(const N2& nd) {
    const float dx = nd.mx[0] - nd.mn[0], dy = nd.mx[1] - nd.mn[1], dz = nd.mx[2] - nd.mn[2];
    return 2.0f * ((dx * dy + dy * dz) + dz * dx);
}

// Greedy candidates of SoftwareBVH4::collapse (software_bvh.hpp:225-247)
// for inner binary node u: open the inner candidate with the largest
// surface area (strict >, first wins) until four.  Returns the count;
// inner[i]: candidate i is an inner binary node.  end, ce: in a pre-order tree,
// the end of u's range and of each candidate's.
__device__ __forceinline__ int greedy_candidates(const rq_bvh2_node* n2, int32_t u, int32_t c[4], bool inner[4],
                                                 int32_t end, int32_t (&ce)[4]) {
    // each candidate's children and surface area, loaded once (slots are
    // static indices, so the records stay in registers)
    int32_t cl[4], cr[4];
    float sa[4];
    auto set = [&](int i, int32_t id, const N2& nd) {
        c[i] = id;
        cl[i] = nd.l;
        cr[i] = nd.r;
        sa[i] = node_area(nd);
    };
    const N2 nd = load_n2(n2, u);
    {
        const N2 a = load_n2(n2, nd.l), b = load_n2(n2, nd.r);
        set(0, nd.l, a);
        set(1, nd.r, b);
    }
    ce[0] = nd.r;
    ce[1] = end;
    ce[2] = ce[3] = 0;
    c[2] = c[3] = -1;
    cl[2] = cl[3] = -1;
    cr[2] = cr[3] = -1;
    sa[2] = sa[3] = 0.0f;
    int nc = 2;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        int best = -1;
        float best_sa = -1.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < nc && cl[i] >= 0 && sa[i] > best_sa) {
                best_sa = sa[i];
                best = i;
            }
        if (best < 0) break;
        int32_t l = 0, r = 0, e = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i == best) {
                l = cl[i];
                r = cr[i];
                e = ce[i];
                ce[i] = r;
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i == nc) ce[i] = e;
        const N2 a = load_n2(n2, l), b = load_n2(n2, r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i == best) set(i, l, a);
            if (i == nc) set(i, r, b);
        }
        ++nc;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) inner[i] = i < nc && cl[i] >= 0;
    return nc;
}

// Writes 4-wide node p from its candidates and the places of the inner ones
// (-1: a leaf).
__device__ __forceinline__ void write_node4(const rq_bvh2_node* n2, const int32_t (&cand)[4], const int32_t (&at)[4],
                                            uint32_t p, rq_bvh4_node* out4, int32_t* map4) {
    float mnx[4], mxx[4], mny[4], mxy[4], mnz[4], mxz[4];
    int32_t ci[4], cc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        mnx[k] = mxx[k] = mny[k] = mxy[k] = mnz[k] = mxz[k] = 0.0f;
        ci[k] = 0;
        cc[k] = 0;
        if (cand[k] >= 0) {
            const N2 nd = load_n2(n2, cand[k]);
            mnx[k] = nd.mn[0];
            mxx[k] = nd.mx[0];
            mny[k] = nd.mn[1];
            mxy[k] = nd.mx[1];
            mnz[k] = nd.mn[2];
            mxz[k] = nd.mx[2];
            if (at[k] >= 0) {
                ci[k] = at[k];
                cc[k] = -1;
            } else {
                ci[k] = nd.l;
                cc[k] = nd.r;
            }
        }
    }
    reinterpret_cast<int4*>(map4)[p] = make_int4(cand[0], cand[1], cand[2], cand[3]);
    float4* o = reinterpret_cast<float4*>(out4 + p);
    o[0] = make_float4(mnx[0], mnx[1], mnx[2], mnx[3]);
    o[1] = make_float4(mxx[0], mxx[1], mxx[2], mxx[3]);
    o[2] = make_float4(mny[0], mny[1], mny[2], mny[3]);
    o[3] = make_float4(mxy[0], mxy[1], mxy[2], mxy[3]);
    o[4] = make_float4(mnz[0], mnz[1], mnz[2], mnz[3]);
    o[5] = make_float4(mxz[0], mxz[1], mxz[2], mxz[3]);
    reinterpret_cast<int4*>(o)[6] = make_int4(ci[0], ci[1], ci[2], ci[3]);
    reinterpret_cast<int4*>(o)[7] = make_int4(cc[0], cc[1], cc[2], cc[3]);
}

// Scratch and outputs of one collapse.
struct CollapseIO {
    const rq_bvh2_node* n2;
    uint32_t* q;        // queue: binary node of each 4-wide node, level by level
    int32_t* cand;      // 4 per queue entry
    int32_t* child_q;   // 4 per queue entry: queue index of inner children, -1
    uint32_t* sz;       // subtree sizes
    uint32_t* par;      // per queue entry: (parent entry << 2) | slot, kNoParent for the root
    unsigned long long* acc;  // per queue entry: (arrived inner children << 32) | their summed sizes
    uint32_t* tail;     // control words: [4..6] per-level append counts, [8..10] hand-over
    rq_bvh4_node* out4;
    int32_t* map4;
};

// Inner children (queue entries) of entry e.
__device__ __forceinline__ uint32_t inner_children(const CollapseIO& io, uint32_t e) {
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) c += __ldcg(io.child_q + 4 * size_t(e) + k) >= 0 ? 1u : 0u;
    return c;
}

// The three phases of the collapse, run by `nthreads` cooperating threads
// (index tid) that meet at `sync()` (false = a barrier gave up; abort):
//   1. top-down per level: candidates, inner candidates appended to q with
//      their parent link;
//   2. subtree sizes bottom-up without level barriers: each entry with no
//      inner children starts a walk; at each parent one 64-bit atomic adds
//      (one arrival, the child's size) and returns the earlier arrivals and
//      sizes, so the arrival that completes the parent carries its size on;
//   3. every entry's pre-order position is the sum over its ancestors of
//      1 + the sizes of the earlier inner siblings (a walk up that stops at
//      the first ancestor whose position a written parent already
//      published), then the node write.
// Block 0 alone expands the top levels while they hold at most NARROW
// entries.  io.tail holds 16 control words.
// Data written inside the collapse is read with ld.cg: other blocks wrote it.
template <uint32_t NARROW, class Sync>
__device__ __forceinline__ bool collapse_levels(const CollapseIO& io, uint32_t tid, uint32_t nthreads,
                                                uint32_t max_levels, Sync sync, uint32_t* err,
                                                uint32_t* total_out, uint32_t* depth_out) {
    const bool root_leaf = load_n2(io.n2, 0).l < 0;
    // Entries of level L+1 are appended at end(L) + an atomic count of their
    // own, io.tail[4 + L % 3]: after the level's sync every thread reads that
    // count while the next level appends to another one, and the one after
    // that is cleared during level L, two syncs after its last reader.
    uint32_t* lvl_cnt = io.tail + 4;
    // Inner candidates take consecutive queue entries: one atomic per warp
    // (the lanes that expand together), each lane's entries after the lower
    // lanes'.  Entry numbers only name queue records; the output does not
    // depend on them.
    auto expand = [&](uint32_t e, uint32_t end, uint32_t depth) {
        const int32_t u = int32_t(__ldcg(io.q + e));
        int32_t c[4] = {-1, -1, -1, -1}, ce[4];
        bool inner[4] = {false, false, false, false};
        if (root_leaf)
            c[0] = 0;
        else
            greedy_candidates(io.n2, u, c, inner, 0, ce);
        const uint32_t cnt = uint32_t(inner[0]) + uint32_t(inner[1]) + uint32_t(inner[2]) + uint32_t(inner[3]);
        const uint32_t act = __activemask();
        const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
        const uint32_t b0 = __ballot_sync(act, cnt & 1u), b1 = __ballot_sync(act, cnt & 2u),
                       b2 = __ballot_sync(act, cnt & 4u);
        const uint32_t below = __popc(b0 & lt) + 2u * __popc(b1 & lt) + 4u * __popc(b2 & lt);
        const uint32_t total = __popc(b0) + 2u * __popc(b1) + 4u * __popc(b2);
        const uint32_t leader = __ffs(act) - 1u;
        uint32_t base = 0;
        if (lane == leader && total) base = atomicAdd(lvl_cnt + depth % 3u, total);
        uint32_t pos = end + __shfl_sync(act, base, leader) + below;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            int32_t cq = -1;
            if (inner[k]) {
                __stcg(io.q + pos, uint32_t(c[k]));
                __stcg(io.par + pos, (e << 2) | uint32_t(k));
                __stcg(io.acc + pos, 0ull);
                cq = int32_t(pos++);
            }
            __stcg(io.cand + 4 * size_t(e) + k, c[k]);
            __stcg(io.child_q + 4 * size_t(e) + k, cq);
        }
    };
    if (tid == 0) {
        __stcg(io.q, 0u);
        __stcg(io.par, kNoParent);
        __stcg(io.acc, 0ull);
        atomicExch(lvl_cnt, 0u);
    }
    if (!sync()) return false;
    uint32_t start = 0, end = 1, depth = 0;
    // the narrow top levels (at most NARROW entries each) by block 0
    // alone, with block barriers; then one sync hands the frontier over
    if (blockIdx.x == 0) {
        while (start < end && end - start <= NARROW && depth + 1 < max_levels) {
            if (threadIdx.x == 0) atomicExch(lvl_cnt + (depth + 1) % 3u, 0u);
            for (uint32_t e = start + threadIdx.x; e < end; e += blockDim.x) expand(e, end, depth);
            __syncthreads();
            const uint32_t n = __ldcg(lvl_cnt + depth % 3u);
            ++depth;
            start = end;
            end += n;
        }
        if (threadIdx.x == 0) {
            __stcg(io.tail + 8, start);
            __stcg(io.tail + 9, end);
            __stcg(io.tail + 10, depth);
        }
    }
    if (!sync()) return false;
    start = __ldcg(io.tail + 8);
    end = __ldcg(io.tail + 9);
    depth = __ldcg(io.tail + 10);
    while (start < end) {
        if (tid == 0) atomicExch(lvl_cnt + (depth + 1) % 3u, 0u);
        for (uint32_t e = start + tid; e < end; e += nthreads) expand(e, end, depth);
        if (!sync()) return false;
        const uint32_t n = __ldcg(lvl_cnt + depth % 3u);
        ++depth;
        start = end;
        end += n;
        if (depth >= max_levels) {
            if (tid == 0) set_err(err, RQ_DERR_QUEUE);
            return false;
        }
    }
    for (uint32_t e = tid; e < end; e += nthreads) {
        if (inner_children(io, e) != 0u) continue;
        uint32_t cur = e, s = 1u;
        __stcg(io.sz + cur, s);
        for (uint32_t guard = 0;; ++guard) {
            const uint32_t pk = __ldcg(io.par + cur);
            if (pk == kNoParent) break;
            if (guard >= max_levels) {
                set_err(err, RQ_DERR_QUEUE);
                break;
            }
            const uint32_t p = pk >> 2;
            const unsigned long long old = atomicAdd(io.acc + p, (1ull << 32) | s);
            if (uint32_t(old >> 32) + 1u < inner_children(io, p)) break;
            s = 1u + uint32_t(old) + s;
            __stcg(io.sz + p, s);
            cur = p;
        }
    }
    if (!sync()) return false;
    // a written node publishes its inner children's positions in `acc`
    // (bit 63 set; phase 2 never sets it), so most walks stop at once
    for (uint32_t e = tid; e < end; e += nthreads) {
        uint32_t pre = 0, cur = e;
        for (;;) {
            const unsigned long long a = __ldcg(io.acc + cur);
            if (a >> 63) {
                pre += uint32_t(a);
                break;
            }
            const uint32_t pk = __ldcg(io.par + cur);
            if (pk == kNoParent) break;  // the root, at 0
            const uint32_t p = pk >> 2, slot = pk & 3u;
            uint32_t off = 1u;
            for (uint32_t j = 0; j < slot; ++j) {
                const int32_t cq = __ldcg(io.child_q + 4 * size_t(p) + j);
                if (cq >= 0) off += __ldcg(io.sz + cq);
            }
            pre += off;
            cur = p;
        }
        uint32_t off = pre + 1u;
        int32_t cand[4], at[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cand[k] = __ldcg(io.cand + 4 * size_t(e) + k);
            const int32_t cq = __ldcg(io.child_q + 4 * size_t(e) + k);
            at[k] = -1;
            if (cq < 0) continue;
            at[k] = int32_t(off);
            __stcg(io.acc + cq, (1ull << 63) | off);
            off += __ldcg(io.sz + cq);
        }
        write_node4(io.n2, cand, at, pre, io.out4, io.map4);
    }
    if (!sync()) return false;
    *total_out = end;
    *depth_out = depth;
    return true;
}

}  // namespace rq
