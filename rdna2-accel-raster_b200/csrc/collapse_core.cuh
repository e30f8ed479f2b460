// collapse_core.cuh — the 4-wide collapse of trees whose binary nodes are in
// depth-first pre-order (every build's), by treelets; shared by k_collapse.cu
// (one tree) and k_forest.cu (all meshes of a batch).
//
// Which binary nodes become 4-wide nodes is decided from the root down, and
// where they go from their subtrees' sizes: level by level over the whole tree
// that was a chain of dependent loads from L2 and a grid barrier per level, at
// 512 threads per SM.  In pre-order a subtree is a range, so here
//   top    one block per tree goes down from the root to the subtrees of at
//          most `limit` binary nodes, the treelets, and lists them;
//   treelets  a block per treelet reads its range once into shared memory and
//          does the levels, sizes and pre-order places there, leaving one
//          16-byte entry per 4-wide node;
//   places one block per tree adds the sizes up and writes the top's nodes;
//   write  the treelets' nodes.
// The result is that of collapse_levels (build_core.cuh), which remains for
// imported trees, whose nodes may lie in any order.  8.3M triangles 460 -> 254
// us (top 45, treelets 100, places 29, write 79), 2.5M with SAH subtrees 160 ->
// 87, 99,225 split at medians 77 -> 40, 512 meshes of 4.73M together (a block per
// mesh before) 261 -> 132.  The two middle steps are chains of short levels; the
// write moves 0.5 GB on 8.3M.  Treelets of at most 1,024 or 512 nodes: 355 and
// 506 us on 8.3M (the top grows); 128, 384 and 512 threads per treelet 102, 144
// and 153 us where 256 take 100.
#pragma once

#include "build_core.cuh"

namespace rq {

constexpr uint32_t kTreeletMax = 2048;   // binary nodes of a treelet at most (34 KB of shared memory)
constexpr uint32_t kCollapseLevels = 120;
constexpr uint32_t kLevelWords = kCollapseLevels + 8;
constexpr uint32_t kTreeletBit = 0x40000000u;
constexpr uint32_t kCollapseT = 256, kTopT = 1024;
constexpr uint32_t kTopChunk = 64;  // top nodes written by a block
constexpr uint32_t kTopRecord = 0xffffffffu;

// One tree's part of a collapse.
struct CollapseTree {
    const rq_bvh2_node* n2;
    rq_bvh4_node* out4;
    int32_t* map4;
    uint32_t* counts;   // [0] binary nodes (in), [1] 4-wide nodes, [2] depth
    // the top's 4-wide nodes: binary node, its range's end (later the node's
    // place), size, candidates, children (-1 none, a top entry, kTreeletBit | treelet)
    uint32_t *q, *end, *size;
    int32_t *cand, *child;
    uint32_t* levels;   // [0] levels of the top (0: the tree is treelet [1]), then their first entries and the end
    uint4* ent;         // by binary node: a treelet's entries from its first node on
};
// The treelets of all trees of a launch.
struct Treelets {
    uint32_t* count;    // zeroed
    uint4* list;        // first node, nodes, level, tree
    uint4* out;         // 4-wide nodes, depth, place
    uint32_t limit;
    uint32_t* err;
};

struct alignas(16) TreeletShared {
    float area[kTreeletMax];
    uint16_t link[kTreeletMax];  // right child; kNone: a leaf
    uint16_t q[kTreeletMax / 2], size[kTreeletMax / 2], pre[kTreeletMax / 2];
    uint16_t cand[kTreeletMax / 2][4], child[kTreeletMax / 2][4];
    uint32_t level[kCollapseLevels + 2];
    uint32_t tail;
    static constexpr uint32_t kNone = 0xffffu;
};

// Down from the root to the treelets (one block).
__device__ __forceinline__ void collapse_top(const CollapseTree& t, uint32_t tree, const Treelets& T) {
    __shared__ uint32_t s_next;
    const uint32_t nodes = t.counts[0];
    if (nodes <= T.limit) {
        if (threadIdx.x == 0) {
            const uint32_t k = atomicAdd(T.count, 1u);
            T.list[k] = make_uint4(0u, nodes, 0u, tree);
            t.levels[0] = 0u;
            t.levels[1] = k;
        }
        return;
    }
    if (threadIdx.x == 0) {
        t.q[0] = 0u;
        t.end[0] = nodes;
        s_next = 1u;
    }
    __syncthreads();
    uint32_t start = 0, end = 1, level = 0;
    while (start < end && level < kCollapseLevels) {
        if (threadIdx.x == 0) t.levels[1 + level] = start;
        for (uint32_t e = start + threadIdx.x; e < end; e += kTopT) {
            int32_t c[4], ce[4];
            bool inner[4];
            greedy_candidates(t.n2, int32_t(t.q[e]), c, inner, int32_t(t.end[e]), ce);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int32_t ch = -1;
                if (inner[k]) {
                    const uint32_t len = uint32_t(ce[k] - c[k]);
                    if (len > T.limit) {
                        const uint32_t at = atomicAdd(&s_next, 1u);
                        t.q[at] = uint32_t(c[k]);
                        t.end[at] = uint32_t(ce[k]);
                        ch = int32_t(at);
                    } else {
                        const uint32_t at = atomicAdd(T.count, 1u);
                        T.list[at] = make_uint4(uint32_t(c[k]), len, level + 1u, tree);
                        ch = int32_t(kTreeletBit | at);
                    }
                }
                t.cand[4 * size_t(e) + k] = c[k];
                t.child[4 * size_t(e) + k] = ch;
            }
        }
        __syncthreads();
        start = end;
        end = s_next;
        ++level;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        t.levels[0] = level;
        t.levels[1 + level] = start;
        if (start < end) {
            set_err(T.err, RQ_DERR_QUEUE);
            // (the entries beyond have no children listed: places skips them)
        }
    }
}

// A treelet's levels, sizes and places (one block).
__device__ __forceinline__ void collapse_treelet(TreeletShared& S, const CollapseTree& t, const Treelets& T,
                                                 uint32_t k, uint4 rec) {
    const uint32_t u = rec.x, len = rec.y;
    for (uint32_t i = threadIdx.x; i < len; i += kCollapseT) {
        const N2 nd = load_n2(t.n2, int32_t(u + i));
        S.link[i] = uint16_t(nd.l < 0 ? TreeletShared::kNone : uint32_t(nd.r) - u);
        S.area[i] = node_area(nd);
    }
    if (threadIdx.x == 0) {
        S.q[0] = 0;
        S.tail = 1u;
    }
    __syncthreads();
    uint32_t depth = 0, start = 0, end = 1;
    bool ok = true;
    while (start < end) {
        if (threadIdx.x == 0) S.level[depth] = start;
        for (uint32_t e = start + threadIdx.x; e < end; e += kCollapseT) {
            const uint32_t v = S.q[e];
            uint32_t c[4] = {v, TreeletShared::kNone, TreeletShared::kNone, TreeletShared::kNone};
            uint32_t right[4] = {S.link[v], TreeletShared::kNone, TreeletShared::kNone, TreeletShared::kNone};
            float sa[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            int nc = 1;
            if (right[0] != TreeletShared::kNone) {  // (the root of a tree of one node is a leaf)
                c[0] = v + 1u;
                c[1] = right[0];
                nc = 2;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    right[i] = S.link[c[i]];
                    sa[i] = S.area[c[i]];
                }
            }
#pragma unroll
            for (int it = 0; it < 2; ++it) {
                int best = -1;
                float best_sa = -1.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < nc && right[i] != TreeletShared::kNone && sa[i] > best_sa) {
                        best_sa = sa[i];
                        best = i;
                    }
                if (best < 0) break;
                uint32_t l = 0, r = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i == best) {
                        l = c[i] + 1u;
                        r = right[i];
                    }
                const uint32_t ll = S.link[l], rl = S.link[r];
                const float la = S.area[l], ra = S.area[r];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i == best) {
                        c[i] = l;
                        right[i] = ll;
                        sa[i] = la;
                    }
                    if (i == nc) {
                        c[i] = r;
                        right[i] = rl;
                        sa[i] = ra;
                    }
                }
                ++nc;
            }
            uint32_t inner = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < nc && right[i] != TreeletShared::kNone) inner |= 1u << i;
            uint32_t at = inner ? atomicAdd(&S.tail, uint32_t(__popc(inner))) : 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t ch = TreeletShared::kNone;
                if ((inner >> i) & 1u) {
                    ch = at++;
                    S.q[ch] = uint16_t(c[i]);
                }
                S.cand[e][i] = uint16_t(i < nc ? c[i] : TreeletShared::kNone);
                S.child[e][i] = uint16_t(ch);
            }
        }
        __syncthreads();
        ++depth;
        start = end;
        end = S.tail;
        __syncthreads();
        if (rec.z + depth >= kCollapseLevels) {
            ok = false;
            break;
        }
    }
    if (!ok) {
        if (threadIdx.x == 0) {
            set_err(T.err, RQ_DERR_QUEUE);
            T.out[k] = make_uint4(0u, depth, 0u, 0u);
        }
        return;
    }
    if (threadIdx.x == 0) S.level[depth] = end;
    __syncthreads();
    for (uint32_t lv = depth; lv-- > 0;) {
        for (uint32_t e = S.level[lv] + threadIdx.x; e < S.level[lv + 1]; e += kCollapseT) {
            uint32_t s = 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = S.child[e][i];
                if (ch != TreeletShared::kNone) s += S.size[ch];
            }
            S.size[e] = uint16_t(s);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        S.pre[0] = 0;
        T.out[k] = make_uint4(end, depth, 0u, 0u);
    }
    __syncthreads();
    for (uint32_t lv = 0; lv < depth; ++lv) {
        for (uint32_t e = S.level[lv] + threadIdx.x; e < S.level[lv + 1]; e += kCollapseT) {
            const uint32_t p = S.pre[e];
            uint32_t off = p + 1u, at[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = S.child[e][i];
                at[i] = 0;  // (no child's place)
                if (ch != TreeletShared::kNone) {
                    at[i] = off;
                    S.pre[ch] = uint16_t(off);
                    off += S.size[ch];
                }
            }
            const uint2 cd = *reinterpret_cast<const uint2*>(S.cand[e]);
            t.ent[u + p] = make_uint4(cd.x, cd.y, at[0] | (at[1] << 16), at[2] | (at[3] << 16));
        }
        __syncthreads();
    }
}

// The sizes and places of the top and of the treelets (one block);
// records for the writing of the top's nodes.
__device__ __forceinline__ void collapse_places(const CollapseTree& t, uint32_t tree, const Treelets& T) {
    __shared__ uint32_t s_depth, s_at;
    const uint32_t levels = t.levels[0];
    if (levels == 0u) {
        if (threadIdx.x == 0) {
            const uint4 o = T.out[t.levels[1]];
            t.counts[1] = o.x;
            t.counts[2] = o.y;
        }
        return;
    }
    const uint32_t all = t.levels[1 + levels], chunks = (all + kTopChunk - 1) / kTopChunk;
    if (threadIdx.x == 0) {
        s_depth = levels;
        s_at = atomicAdd(T.count, chunks);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < chunks; i += kTopT)
        T.list[s_at + i] = make_uint4(i * kTopChunk, min(kTopChunk, all - i * kTopChunk), kTopRecord, tree);
    auto size_of = [&](int32_t ch) {
        if (uint32_t(ch) & kTreeletBit) return T.out[uint32_t(ch) & ~kTreeletBit].x;
        return uint32_t(ch) < all ? t.size[ch] : 0u;
    };
    for (uint32_t lv = levels; lv-- > 0;) {
        for (uint32_t e = t.levels[1 + lv] + threadIdx.x; e < t.levels[2 + lv]; e += kTopT) {
            uint32_t s = 1;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int32_t ch = t.child[4 * size_t(e) + k];
                if (ch >= 0) s += size_of(ch);
                if (ch >= 0 && (uint32_t(ch) & kTreeletBit))
                    atomicMax(&s_depth, lv + 1u + T.out[uint32_t(ch) & ~kTreeletBit].y);
            }
            t.size[e] = s;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        t.end[0] = 0u;  // (the root's place)
        t.counts[1] = t.size[0];
        t.counts[2] = s_depth;
    }
    __syncthreads();
    for (uint32_t lv = 0; lv < levels; ++lv) {
        for (uint32_t e = t.levels[1 + lv] + threadIdx.x; e < t.levels[2 + lv]; e += kTopT) {
            uint32_t off = t.end[e] + 1u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int32_t ch = t.child[4 * size_t(e) + k];
                if (ch < 0) continue;
                if (uint32_t(ch) & kTreeletBit)
                    T.out[uint32_t(ch) & ~kTreeletBit].z = off;
                else if (uint32_t(ch) < all)
                    t.end[ch] = off;
                off += size_of(ch);
            }
        }
        __syncthreads();
    }
}

// v[j] of lane k of a quad becomes v[k] of its lane j.
__device__ __forceinline__ void quad_transpose(float (&v)[4], uint32_t k) {
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        const float r = __shfl_xor_sync(0xffffffffu, k & 1u ? v[i] : v[i + 1], 1);
        (k & 1u ? v[i] : v[i + 1]) = r;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float r = __shfl_xor_sync(0xffffffffu, k & 2u ? v[i] : v[i + 2], 2);
        (k & 2u ? v[i] : v[i + 2]) = r;
    }
}

// The nodes of a record, a quad of lanes each: a lane reads one candidate and
// writes two of the node's eight rows, so that a node leaves as two pieces of
// 64 bytes (a thread per node wrote eight pieces of 16: 122 us for 61).
__device__ __forceinline__ void collapse_write(const CollapseTree& t, const Treelets& T, uint32_t rec_at, uint4 rec) {
    const bool top = rec.z == kTopRecord;
    const uint4 out = top ? make_uint4(rec.y, 0u, 0u, 0u) : T.out[rec_at];
    const uint32_t k = threadIdx.x & 3u;
    for (uint32_t i0 = 0; i0 < out.x; i0 += kCollapseT / 4) {
        const uint32_t i = i0 + threadIdx.x / 4u;
        const bool on = i < out.x;
        int32_t c = -1, at = -1;
        uint32_t p = 0;
        if (on && top) {
            const uint32_t e = rec.x + i;
            p = t.end[e];
            c = t.cand[4 * size_t(e) + k];
            const int32_t ch = t.child[4 * size_t(e) + k];
            if (ch >= 0) at = int32_t(uint32_t(ch) & kTreeletBit ? T.out[uint32_t(ch) & ~kTreeletBit].z : t.end[ch]);
        } else if (on) {
            p = out.z + i;
            const uint32_t* e = reinterpret_cast<const uint32_t*>(t.ent + rec.x + i) + (k >> 1);
            const uint32_t sh = 16u * (k & 1u), cw = (e[0] >> sh) & 0xffffu, aw = (e[2] >> sh) & 0xffffu;
            if (cw != TreeletShared::kNone) c = int32_t(rec.x + cw);
            if (aw) at = int32_t(out.z + aw);
        }
        float lo[4] = {0.0f, 0.0f, 0.0f, 0.0f}, hi[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // rows 0..3, 4..7
        if (c >= 0) {
            const N2 nd = load_n2(t.n2, c);
            lo[0] = nd.mn[0];
            lo[1] = nd.mx[0];
            lo[2] = nd.mn[1];
            lo[3] = nd.mx[1];
            hi[0] = nd.mn[2];
            hi[1] = nd.mx[2];
            hi[2] = __int_as_float(at >= 0 ? at : nd.l);
            hi[3] = __int_as_float(at >= 0 ? -1 : nd.r);
        }
        quad_transpose(lo, k);
        quad_transpose(hi, k);
        if (on) {
            float4* o = reinterpret_cast<float4*>(t.out4 + p);
            o[k] = make_float4(lo[0], lo[1], lo[2], lo[3]);
            o[4 + k] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            t.map4[4 * size_t(p) + k] = c;
        }
    }
}

// Trees: trees(k) is tree k.
template <class Trees>
__global__ void __launch_bounds__(kTopT) k_collapse_top(const __grid_constant__ Trees trees,
                                                             const __grid_constant__ Treelets T) {
    collapse_top(trees(blockIdx.x), blockIdx.x, T);
}
template <class Trees>
__global__ void __launch_bounds__(kCollapseT) k_collapse_treelets(const __grid_constant__ Trees trees,
                                                                  const __grid_constant__ Treelets T) {
    __shared__ TreeletShared S;
    const uint32_t n = *T.count;
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const uint4 rec = T.list[k];
        collapse_treelet(S, trees(rec.w), T, k, rec);
        __syncthreads();
    }
}
template <class Trees>
__global__ void __launch_bounds__(kTopT) k_collapse_places(const __grid_constant__ Trees trees,
                                                                const __grid_constant__ Treelets T) {
    collapse_places(trees(blockIdx.x), blockIdx.x, T);
}
template <class Trees>
__global__ void __launch_bounds__(kCollapseT) k_collapse_write(const __grid_constant__ Trees trees,
                                                               const __grid_constant__ Treelets T) {
    const uint32_t n = *T.count;
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const uint4 rec = T.list[k];
        collapse_write(trees(rec.w), T, k, rec);
    }
}

template <class Trees>
void launch_collapse(const Trees& trees, const Treelets& T, uint32_t count, int sms, cudaStream_t st) {
    k_collapse_top<<<count, kTopT, 0, st>>>(trees, T);
    k_collapse_treelets<<<uint32_t(sms) * 6u, kCollapseT, 0, st>>>(trees, T);
    k_collapse_places<<<count, kTopT, 0, st>>>(trees, T);
    k_collapse_write<<<uint32_t(sms) * 8u, kCollapseT, 0, st>>>(trees, T);
}

}  // namespace rq
