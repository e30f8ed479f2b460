// k_forest.cu — the LBVH builds of all meshes of a batch together: every step
// of k_build.cu runs once over all of them, its blocks dealt out by tables
// made when the batch is created (no block spans two meshes), with each mesh's
// arrays at its own offset.  The per-element steps are build_core.cuh's, so
// every mesh's bytes equal a separate rq_build of that mesh.
//
// A build by one block or cluster per mesh, the form this replaces, was bound
// by the largest meshes' chains of steps on one SM: 2.06 ms for 512 meshes of
// 64 to 65,536 triangles (4.73M).  All meshes together take 0.80 ms: the tree
// 0.28, the sort 0.22, the collapse 0.13, the node writes 0.07.
// Batches of more than kGroupTris triangles go in groups of whole meshes that
// use the scratch in turn.
#include <algorithm>
#include <numeric>
#include <vector>

#include "build_core.cuh"
#include "collapse_core.cuh"
#include "rq_batch.h"
#include "rq_device.cuh"
#include "rq_internal.h"

namespace {

using namespace rq;

constexpr int kT = 256;
constexpr uint32_t kGroupTris = 16u << 20;
static_assert(kTreeLeaves % kT == 0, "a block of elements is a block of leaves");

struct ForestScratch {
    float4* cent;
    uint32_t* zero;     // zeroed per build, from here ...
    uint32_t* bounds;   // 6 per mesh: maxima of f2o, of ~f2o
    uint32_t* misc;     // [0] unfinished nodes, [1] scan ticket, [2] treelets
    size_t zero_bytes;  // ... to here
    uint32_t *keys[2], *vals[2];
    uint32_t* counts;   // sort: 256 per tile
    float4 *rec, *leaf, *slot;
    uint16_t* ch;
    uint32_t *seen, *a, *scan_status;
    uint2* top_list;
    uint32_t* q;
    int32_t *cand, *child_q;
    uint32_t *sz, *end, *levels;
};

size_t carve(void* base, const rq_forest_group& g, ForestScratch& s) {
    Carve c{reinterpret_cast<uintptr_t>(base), 0};
    const size_t N = g.tris;
    s.bounds = c.take<uint32_t>(6ull * g.segs);
    s.misc = c.take<uint32_t>(16);
    s.seen = c.take<uint32_t>(g.seen_words);
    s.zero = s.bounds;
    s.zero_bytes = c.off;
    s.cent = c.take<float4>(N);
    for (int k = 0; k < 2; ++k) s.keys[k] = c.take<uint32_t>(N);
    for (int k = 0; k < 2; ++k) s.vals[k] = c.take<uint32_t>(N);
    s.counts = c.take<uint32_t>(256ull * g.tiles);
    s.rec = c.take<float4>(2 * N);
    s.leaf = c.take<float4>(2 * N);
    s.slot = c.take<float4>(2 * N);
    s.ch = c.take<uint16_t>(N);
    s.a = c.take<uint32_t>(N);
    s.scan_status = c.take<uint32_t>(rq_scan_tiles(uint32_t(N)) + 1);
    s.top_list = c.take<uint2>(N);
    s.q = c.take<uint32_t>(N);
    s.cand = c.take<int32_t>(4 * N);
    s.child_q = c.take<int32_t>(4 * N);
    s.sz = c.take<uint32_t>(N);
    s.end = c.take<uint32_t>(N);
    s.levels = c.take<uint32_t>(size_t(kLevelWords) * g.segs);
    return c.off + 256;
}

struct ForestArgs {
    const float* pos;
    uint32_t sf;
    const uint32_t* idx;
    uint32_t max_leaf;
    const rq_forest_seg* segs;
    const uint2* blocks;   // (segment, first element)
    rq_bvh2_node* nodes2;
    rq_triangle* tris;
    uint32_t *perm, *skeys;
    rq_bvh4_node* nodes4;
    int32_t* map4;
    uint32_t* counts;      // 4 per mesh
    uint32_t* err;
    ForestScratch s;
};

__global__ void __launch_bounds__(kT) k_forest_centroids(const __grid_constant__ ForestArgs A) {
    __shared__ float s_red[6][kT / 32];
    const uint2 b = A.blocks[blockIdx.x];
    const rq_forest_seg g = A.segs[b.x];
    float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    const uint32_t end = min(b.y + kTreeLeaves, g.n);
    for (uint32_t i = b.y + threadIdx.x; i < end; i += kT) {
        F3 p0, p1, p2;
        load_tri(A.pos + size_t(g.vert) * A.sf, A.sf, A.idx + 3ull * g.tri, i, p0, p1, p2);
        const float4 c = centroid(p0, p1, p2);
        A.s.cent[g.first + i] = c;
        const float x[3] = {c.x, c.y, c.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = fminf(v[k], x[k]);
            v[3 + k] = fmaxf(v[3 + k], x[k]);
        }
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float y = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = k < 3 ? fminf(v[k], y) : fmaxf(v[k], y);
        }
        if (lane == 0) s_red[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const uint32_t k = threadIdx.x;
        float r = s_red[k][0];
        for (int w = 1; w < kT / 32; ++w) r = k < 3 ? fminf(r, s_red[k][w]) : fmaxf(r, s_red[k][w]);
        atomicMax(A.s.bounds + 6ull * b.x + k, k < 3 ? ~f2o(r) : f2o(r));
    }
}

__global__ void __launch_bounds__(kT) k_forest_morton(const __grid_constant__ ForestArgs A) {
    const uint2 b = A.blocks[blockIdx.x];
    const rq_forest_seg g = A.segs[b.x];
    const uint32_t* bd = A.s.bounds + 6ull * b.x;
    const float lx = o2f(~bd[0]), ly = o2f(~bd[1]), lz = o2f(~bd[2]);
    const float scale = morton_scale(lx, ly, lz, o2f(bd[3]), o2f(bd[4]), o2f(bd[5]));
    const uint32_t end = min(b.y + kTreeLeaves, g.n);
    for (uint32_t i = b.y + threadIdx.x; i < end; i += kT) {
        A.s.keys[0][g.first + i] = morton30(A.s.cent[g.first + i], lx, ly, lz, scale);
        A.s.vals[0][g.first + i] = i;
    }
}

// A mesh's part of the tree arrays.
__device__ __forceinline__ TreeOut tree_of(const ForestArgs& A, const rq_forest_seg& g) {
    const size_t o = g.first;
    return TreeOut{A.tris + g.tri,    A.perm + g.tri,    A.skeys + g.tri,   A.s.ch + o,
                   A.s.rec + 2 * o,   A.s.leaf + 2 * o,  A.s.slot + 2 * o,  A.s.seen + g.seen};
}

__global__ void __launch_bounds__(kTreeT, kTreeBlocks) k_forest_tree(const __grid_constant__ ForestArgs A) {
    __shared__ TreeShared S;
    const uint2 b = A.blocks[blockIdx.x];
    const rq_forest_seg g = A.segs[b.x];
    tree_climb_block(S, b.y, g.n, A.pos + size_t(g.vert) * A.sf, A.sf, A.idx + 3ull * g.tri, A.max_leaf,
                     A.s.keys[0] + g.first, A.s.vals[0] + g.first, tree_of(A, g));
    if (threadIdx.x == 0 && S.count) S.base = atomicAdd(A.s.misc, S.count);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < S.count; i += kTreeT)
        A.s.top_list[S.base + i] = make_uint2(b.x, 2u * b.y + S.list[i]);
}

__global__ void __launch_bounds__(kT) k_forest_tree_top(const __grid_constant__ ForestArgs A) {
    const uint32_t m = A.s.misc[0];
    for (uint32_t j = blockIdx.x * kT + threadIdx.x; j < m; j += gridDim.x * kT) {
        const uint2 w = A.s.top_list[j];
        const rq_forest_seg g = A.segs[w.x];
        tree_climb_top(w.y, g.n, A.max_leaf, A.s.keys[0] + g.first, tree_of(A, g));
    }
}

// The scan of the emission counts over all meshes, from a mesh's start on.
struct ScanFrom {
    const uint32_t* a;
    uint32_t base;
    __device__ uint32_t operator[](uint32_t i) const { return a[i] - base; }
};

__global__ void __launch_bounds__(kT) k_forest_emit(const __grid_constant__ ForestArgs A) {
    const uint2 b = A.blocks[blockIdx.x];
    const rq_forest_seg g = A.segs[b.x];
    const TreeOut out = tree_of(A, g);
    const ScanFrom scan{A.s.a + g.first, A.s.a[g.first]};
    const uint32_t end = min(b.y + kTreeLeaves, g.n);
    for (uint32_t p = b.y + threadIdx.x; p < end; p += kT) {
        const uint32_t total = tree_write(p, out, scan, A.nodes2 + 2ull * g.tri);
        if (p == g.n - 1) {
            A.counts[4ull * g.mesh] = total;
            A.counts[4ull * g.mesh + 3] = A.max_leaf;
        }
    }
}

// The meshes as the collapse sees them.
struct ForestTrees {
    ForestArgs A;
    __device__ CollapseTree operator()(uint32_t seg) const {
        const rq_forest_seg g = A.segs[seg];
        const size_t o = g.first;
        return CollapseTree{A.nodes2 + 2ull * g.tri, A.nodes4 + g.tri,   A.map4 + 4ull * g.tri, A.counts + 4ull * g.mesh,
                            A.s.q + o,               A.s.end + o,        A.s.sz + o,            A.s.cand + 4 * o,
                            A.s.child_q + 4 * o,     A.s.levels + size_t(kLevelWords) * seg,
                            reinterpret_cast<uint4*>(A.s.rec) + 2 * o};
    }
};
}  // namespace

void rq_forest_plan(const std::vector<rq_mesh_desc>& meshes, rq_forest& f) {
    std::vector<uint32_t> by_place(meshes.size());
    std::iota(by_place.begin(), by_place.end(), 0u);
    std::sort(by_place.begin(), by_place.end(),
              [&](uint32_t a, uint32_t b) { return meshes[a].triangle_offset < meshes[b].triangle_offset; });
    rq_forest_group g{};
    auto close = [&] {
        if (!g.segs) return;
        f.seg_tiles.push_back(g.tiles);
        f.groups.push_back(g);
    };
    for (uint32_t m : by_place) {
        const rq_mesh_desc& d = meshes[m];
        if (!g.segs || g.tris + d.num_triangles > kGroupTris) {
            close();
            g = rq_forest_group{};
            g.seg0 = uint32_t(f.segs.size());
            g.block0 = uint32_t(f.blocks.size());
            g.tile0 = uint32_t(f.tiles.size());
            g.begin0 = uint32_t(f.seg_tiles.size());
        }
        f.segs.push_back(rq_forest_seg{g.tris, d.triangle_offset, d.vertex_offset, d.num_triangles, m, g.seen_words});
        g.seen_words += d.num_triangles / 32 + 1;
        for (uint32_t i = 0; i < d.num_triangles; i += kTreeLeaves, ++g.blocks) f.blocks.push_back(make_uint2(g.segs, i));
        f.seg_tiles.push_back(g.tiles);
        for (uint32_t i = 0; i < d.num_triangles; i += RQ_SORT_TILE, ++g.tiles)
            f.tiles.push_back(rq_sort_tile{g.tris + i, std::min(RQ_SORT_TILE, d.num_triangles - i), g.tris, 0u});
        ++g.segs;
        g.tris += d.num_triangles;
    }
    close();
}

size_t rq_forest_scratch_bytes(const rq_forest& f) {
    size_t most = 0;
    ForestScratch s;
    for (const rq_forest_group& g : f.groups) most = std::max(most, carve(nullptr, g, s));
    return most;
}

int rq_launch_batch_build(rq_ctx* ctx, rq_batch* b, const float* pos, uint32_t stride_bytes, const uint32_t* idx,
                          cudaStream_t st) {
    const rq_forest& f = b->forest;
    for (const rq_forest_group& g : f.groups) {
        ForestArgs a;
        carve(b->scratch, g, a.s);
        a.pos = pos;
        a.sf = stride_bytes / 4;
        a.idx = idx;
        a.max_leaf = b->max_leaf;
        a.segs = f.d_segs + g.seg0;
        a.blocks = f.d_blocks + g.block0;
        a.nodes2 = b->nodes2;
        a.tris = b->tris;
        a.perm = b->perm;
        a.skeys = b->skeys;
        a.nodes4 = b->nodes4;
        a.map4 = b->map4;
        a.counts = b->d_counts;
        a.err = ctx->d_err;
        cudaError_t e = cudaMemsetAsync(a.s.zero, 0, a.s.zero_bytes, st);
        if (e != cudaSuccess) return rq_cuda_status(ctx, e, "batch build scratch");
        k_forest_centroids<<<g.blocks, kT, 0, st>>>(a);
        k_forest_morton<<<g.blocks, kT, 0, st>>>(a);
        const SortIO io{{a.s.keys[0], a.s.keys[1]}, {a.s.vals[0], a.s.vals[1]}, 0, a.s.counts};
        int rb = 0;
        int rc = rq_launch_sort_tiles(ctx, io, f.d_tiles + g.tile0, g.tiles, f.d_seg_tiles + g.begin0, g.segs, 30, st,
                                      &rb);
        if (rc) return rc;
        if (rb != 0) return rq_set_error(ctx, RQ_ERR_STATE, "sorted keys in the other buffer");
        k_forest_tree<<<g.blocks, kTreeT, 0, st>>>(a);
        k_forest_tree_top<<<uint32_t(ctx->num_sms) * 4u, kT, 0, st>>>(a);
        rq_launch_scan(ctx, a.s.ch, a.s.a, g.tris, a.s.scan_status, a.s.misc + 1, st);
        k_forest_emit<<<g.blocks, kT, 0, st>>>(a);
        // (the tree's records and the centroids are free by now)
        launch_collapse(ForestTrees{a},
                        Treelets{a.s.misc + 2, reinterpret_cast<uint4*>(a.s.cent), reinterpret_cast<uint4*>(a.s.leaf),
                                 kTreeletMax, a.err},
                        g.segs, ctx->num_sms, st);
        e = cudaGetLastError();
        if (e != cudaSuccess) return rq_cuda_status(ctx, e, "batch build launch");
    }
    return RQ_OK;
}
