// rq_batch.h — host-side state of a batch handle (many meshes, one
// allocation) and the launchers of k_batch.cu and k_forest.cu.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "rq_internal.h"

// One mesh in a group of meshes built together: where its elements lie in the
// scratch arrays, its descriptor's offsets, its triangles, its number, its
// first word of arrival bits.
struct rq_forest_seg {
    uint32_t first, tri, vert, n, mesh, seen;
};
struct rq_forest_group {
    uint32_t seg0 = 0, segs = 0;      // segments (meshes)
    uint32_t block0 = 0, blocks = 0;  // element blocks
    uint32_t tile0 = 0, tiles = 0;    // sort tiles
    uint32_t begin0 = 0;              // first tile of each segment, and the end: segs + 1 entries
    uint32_t tris = 0;
    uint32_t seen_words = 0;          // arrival bits, a whole number of words per segment
};
// The tables that deal a batch's builds out to blocks (k_forest.cu).
struct rq_forest {
    std::vector<rq_forest_group> groups;
    std::vector<rq_forest_seg> segs;
    std::vector<uint2> blocks;        // (segment in the group, first element)
    std::vector<rq_sort_tile> tiles;
    std::vector<uint32_t> seg_tiles;
    rq_forest_seg* d_segs = nullptr;
    uint2* d_blocks = nullptr;
    rq_sort_tile* d_tiles = nullptr;
    uint32_t* d_seg_tiles = nullptr;
};
void rq_forest_plan(const std::vector<rq_mesh_desc>& meshes, rq_forest& f);
size_t rq_forest_scratch_bytes(const rq_forest& f);

struct rq_batch {
    rq_ctx* ctx = nullptr;
    int device = 0;
    uint32_t num_meshes = 0;
    uint32_t total_tris = 0;
    uint32_t max_leaf = 4;
    std::vector<rq_mesh_desc> meshes;  // host copy
    // arrays of all meshes: mesh m's binary nodes start at 2*triangle_offset,
    // its triangles / permutation / keys / 4-wide nodes at triangle_offset
    void* mem = nullptr;
    size_t mem_bytes = 0;
    rq_bvh2_node* nodes2 = nullptr;
    rq_triangle* tris = nullptr;
    uint32_t* perm = nullptr;
    uint32_t* skeys = nullptr;
    rq_bvh4_node* nodes4 = nullptr;
    int32_t* map4 = nullptr;
    uint32_t* d_counts = nullptr;  // 4 per mesh: nodes2, nodes4, depth4, max leaf
    rq_mesh_desc* d_meshes = nullptr;
    rq_forest forest;              // how the builds are dealt out
    void* scratch = nullptr;       // build scratch, sized for the largest group
    uint32_t build_slices = 0;     // reported as max_build_blocks
    rq_batch_tuning tune{};        // launch shapes
    std::vector<uint32_t> h_counts;
    bool counts_valid = false;
    uint32_t max_depth = 0;
    bool built = false;
    cudaStream_t last_stream = nullptr;
};

// Whether a traversal kernel exists for this shape.
bool rq_batch_trace_shape_ok(uint32_t threads, uint32_t chunk, uint32_t regs);
int rq_launch_batch_build(rq_ctx* ctx, rq_batch* b, const float* pos, uint32_t stride_bytes, const uint32_t* idx,
                          cudaStream_t st);
int rq_launch_batch_trace(rq_ctx* ctx, const rq_batch* b, const rq_ray* rays, const uint32_t* ray_mesh,
                          const uint32_t* ray_flags, uint32_t n, uint32_t flags, rq_hit* hits, rq_ray_stats* stats,
                          uint32_t* ctr, cudaStream_t st);
