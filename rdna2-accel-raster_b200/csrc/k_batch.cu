// k_batch.cu — one persistent traversal launch over the rays of all meshes of
// a batch (trace_engine.cuh with per-ray BVH and per-ray any hit).  The builds
// are k_forest.cu's.
#include <algorithm>

#include "rq_batch.h"
#include "rq_device.cuh"
#include "rq_internal.h"
#include "trace_engine.cuh"

namespace {

// ------------------------------------------------------------------ trace
template <bool STATS>
struct BatchSrc {
    static constexpr bool kMulti = true;
    struct Meta {
        const uint32_t* perm;
    };
    uint32_t total;
    const rq_ray* rays;
    const uint32_t* ray_mesh;
    const uint32_t* ray_flags;
    uint32_t flags;
    const rq_mesh_desc* meshes;
    const rq_bvh4_node* nodes4;
    const rq_triangle* tris;
    const uint32_t* perm;
    rq_hit* hits;
    rq_ray_stats* stats;

    __device__ bool make(uint32_t id, rq::Ray& r, Meta& m) const {
        const float4* rp = reinterpret_cast<const float4*>(rays + id);
        const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
        const size_t toff = __ldg(&meshes[__ldg(ray_mesh + id)].triangle_offset);
        r.o = rq::F3{r0.x, r0.y, r0.z};
        r.d = rq::F3{r1.x, r1.y, r1.z};
        r.tmin = r0.w;
        r.tmax = r1.w;
        r.nodes = nodes4 + toff;
        r.tris = tris + toff;
        r.any = ((ray_flags ? __ldg(ray_flags + id) : flags) & RQ_TRACE_ANY) != 0u;
        m.perm = perm + toff;
        return true;
    }

    __device__ void finish(uint32_t id, const Meta& m, const rq::Ray&, const rq::Hit& h) const {
        uint4 out = make_uint4(0u, __float_as_uint(-1.0f), 0xffffffffu, 0xffffffffu);
        if (h.hit) out = make_uint4(1u, __float_as_uint(h.t), 0u, __ldg(m.perm + h.idx));
        reinterpret_cast<uint4*>(hits)[id] = out;
        if (STATS) reinterpret_cast<uint4*>(stats)[id] = make_uint4(h.hit ? 1u : 0u, h.boxes, h.tris, 0u);
    }
};

// Traversal blocks of TT threads, ray ids taken CHUNK at a time, and (REGS)
// launch bounds that hold registers to REGS per thread: the tuned shapes.
// The stack has `rows` entries per lane (from the batch's deepest tree; 32 bits
// name every node of a mesh of at most 2^20 triangles); idle lanes are refilled
// once `refill_min` of a warp's lanes are idle.
template <bool MT, bool STATS, int TT, int CHUNK, int REGS>
__global__ void __launch_bounds__(TT, 65536 / (TT * (REGS ? REGS : 65536 / TT)))
    k_batch_trace(const __grid_constant__ BatchSrc<STATS> src, uint32_t* ctr, uint32_t* err, int rows,
                  int refill_min) {
    extern __shared__ __align__(16) uint32_t s_entries[];
    rq::trace_persistent<rq::kAnyPerRay, MT, STATS, TT, const BatchSrc<STATS>, CHUNK>(
        nullptr, nullptr, src, ctr, s_entries + threadIdx.x, rows, err, refill_min);
}

// Kernel of a traversal shape (only the default shape has the counting and
// reference-arithmetic variants).
template <bool MT, bool STATS>
const void* trace_kernel(uint32_t tt, uint32_t chunk, uint32_t regs) {
#define RQ_SHAPE(T, C, R) \
    if (tt == T && chunk == C && regs == R) return reinterpret_cast<const void*>(k_batch_trace<MT, STATS, T, C, R>);
#define RQ_SHAPES(T, C) RQ_SHAPE(T, C, 0) RQ_SHAPE(T, C, 64) RQ_SHAPE(T, C, 80)
    if constexpr (!MT && !STATS) {
        RQ_SHAPES(64, 32) RQ_SHAPES(64, 64) RQ_SHAPES(128, 64) RQ_SHAPES(256, 32) RQ_SHAPES(256, 64)
        RQ_SHAPE(128, 32, 64) RQ_SHAPE(128, 32, 80)
        // a budget of 72 registers: 7 blocks of 128 (14 of 64) threads per SM
        RQ_SHAPE(64, 32, 72) RQ_SHAPE(64, 64, 72) RQ_SHAPE(128, 32, 72) RQ_SHAPE(128, 64, 72)
    }
    RQ_SHAPE(128, 32, 0)
#undef RQ_SHAPES
#undef RQ_SHAPE
    return nullptr;
}

}  // namespace

bool rq_batch_trace_shape_ok(uint32_t threads, uint32_t chunk, uint32_t regs) {
    return trace_kernel<false, false>(threads, chunk, regs) != nullptr;
}

int rq_launch_batch_trace(rq_ctx* ctx, const rq_batch* b, const rq_ray* rays, const uint32_t* ray_mesh,
                          const uint32_t* ray_flags, uint32_t n, uint32_t flags, rq_hit* hits, rq_ray_stats* stats,
                          uint32_t* ctr, cudaStream_t st) {
    const uint32_t bound = 3u * (b->max_depth + 2u) + 1u;
    if (bound > 128u) return rq_set_error(ctx, RQ_ERR_UNSUPPORTED, "4-wide tree deeper than 40 levels");
    const bool mt = flags & RQ_TRI_MT;
    // the counting and reference-arithmetic variants run in the default shape
    const bool tuned = !mt && !stats;
    const uint32_t tt = tuned ? b->tune.trace_threads : 128u;
    const uint32_t chunk = tuned ? b->tune.trace_chunk : 32u;
    const uint32_t regs = tuned ? b->tune.trace_reg_cap : 0u;
    int refill_min = int(tuned && b->tune.trace_refill_min ? b->tune.trace_refill_min : 1u);
    // for the deepest tree, or for the tree the tuned entry count (3 per level)
    // was chosen for
    int rows = rq::rebuild_rows((std::max(bound, b->tune.stack_entries) + 2u) / 3u - 3u);
    const void* kern = mt ? (stats ? trace_kernel<true, true>(tt, chunk, regs) : trace_kernel<true, false>(tt, chunk, regs))
                          : (stats ? trace_kernel<false, true>(tt, chunk, regs) : trace_kernel<false, false>(tt, chunk, regs));
    if (!kern) return rq_set_error(ctx, RQ_ERR_INVALID_ARG, "no traversal kernel for this shape");
    const size_t smem = size_t(rows) * tt * sizeof(uint32_t);
    cudaError_t e = cudaMemsetAsync(ctr, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess && smem > 48 * 1024)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, int(tt), smem);
    if (e == cudaSuccess) {
        if (b->tune.trace_blocks_per_sm && int(b->tune.trace_blocks_per_sm) < per_sm)
            per_sm = int(b->tune.trace_blocks_per_sm);
        uint32_t blocks = uint32_t(ctx->num_sms) * uint32_t(per_sm > 0 ? per_sm : 1);
        blocks = std::max(1u, std::min(blocks, (n + tt - 1) / tt));
        uint32_t* err = ctx->d_err;
        if (stats) {
            BatchSrc<true> src{n, rays, ray_mesh, ray_flags, flags, b->d_meshes, b->nodes4, b->tris, b->perm, hits,
                               stats};
            void* args[] = {&src, &ctr, &err, &rows, &refill_min};
            e = cudaLaunchKernel(kern, dim3(blocks), dim3(tt), args, smem, st);
        } else {
            BatchSrc<false> src{n, rays, ray_mesh, ray_flags, flags, b->d_meshes, b->nodes4, b->tris, b->perm, hits,
                                nullptr};
            void* args[] = {&src, &ctr, &err, &rows, &refill_min};
            e = cudaLaunchKernel(kern, dim3(blocks), dim3(tt), args, smem, st);
        }
    }
    return rq_cuda_status(ctx, e, "batch trace launch");
}
