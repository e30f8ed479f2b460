// Host-side check of the uploads in capi_batch.cpp and tlas.cpp against a model
// of CUDA's ordering rules (no GPU): a host-to-device cudaMemcpy from pageable
// memory and a cudaMemset return once they are queued on the legacy stream,
// and a non-blocking stream does not wait for that stream.  Every write is kept
// until the stream it is queued on is synchronised or a kernel of that same
// stream follows; the launchers below take what a kernel would read.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "rq_batch.h"
#include "rq_tlas.h"

namespace {
struct Write {
    cudaStream_t stream;
    const char *begin, *end;
};
std::vector<Write> pending;
int failures = 0;

cudaError_t queue(cudaStream_t st, void* to, size_t n) {
    pending.push_back({st, static_cast<char*>(to), static_cast<char*>(to) + n});
    return cudaSuccess;
}
// A kernel on `st` reads [p, p + n).
void reads(cudaStream_t st, const void* p, size_t n, const char* what) {
    const char* b = static_cast<const char*>(p);
    for (const Write& w : pending)
        if (w.stream != st && w.begin < b + n && b < w.end) {
            std::printf("%s may be read before it is written\n", what);
            ++failures;
            return;
        }
}
}  // namespace

// ------------------------------------------------------------ CUDA runtime
extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::calloc(1, n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind k) {
    std::memcpy(to, from, n);
    return k == cudaMemcpyHostToDevice ? queue(nullptr, to, n) : cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::memcpy(to, from, n);
    return queue(st, to, n);
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
    std::memset(p, v, n);
    return queue(nullptr, p, n);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    std::memset(p, v, n);
    return queue(st, p, n);
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    std::vector<Write> left;
    for (const Write& w : pending)
        if (w.stream != st) left.push_back(w);
    pending = left;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    pending.clear();
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaErrorUnknown; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaErrorUnknown; }
}

// ------------------------------------------------- the rest of the library
int rq_set_error(rq_ctx*, int status, const std::string&) { return status; }
int rq_cuda_status(rq_ctx*, cudaError_t e, const char*) { return e == cudaSuccess ? RQ_OK : RQ_ERR_CUDA; }
bool rq_batch_trace_shape_ok(uint32_t, uint32_t, uint32_t) { return true; }
size_t rq_forest_scratch_bytes(const rq_forest&) { return 256; }
void rq_forest_plan(const std::vector<rq_mesh_desc>& meshes, rq_forest& f) {
    f.segs.resize(meshes.size());
    f.blocks.resize(3);
    f.tiles.resize(2);
    f.seg_tiles.resize(meshes.size() + 1);
    f.groups.resize(1);
}
int rq_launch_batch_build(rq_ctx*, rq_batch* b, const float*, uint32_t, const uint32_t*, cudaStream_t st) {
    const rq_forest& f = b->forest;
    reads(st, b->d_meshes, sizeof(rq_mesh_desc) * b->num_meshes, "the batch's mesh table");
    reads(st, f.d_segs, sizeof(rq_forest_seg) * b->num_meshes, "the batch's segment table");
    reads(st, f.d_blocks, sizeof(uint2) * 3, "the batch's block table");
    reads(st, f.d_tiles, sizeof(rq_sort_tile) * 2, "the batch's sort tiles");
    reads(st, f.d_seg_tiles, sizeof(uint32_t) * (b->num_meshes + 1), "the batch's tile starts");
    reads(st, b->d_counts, sizeof(uint32_t) * 4 * b->num_meshes, "the batch's counts");
    return RQ_OK;
}
int rq_launch_batch_trace(rq_ctx*, const rq_batch*, const rq_ray*, const uint32_t*, const uint32_t*, uint32_t, uint32_t,
                          rq_hit*, rq_ray_stats*, uint32_t*, cudaStream_t) {
    return RQ_OK;
}
int rq_launch_instance_boxes(rq_ctx*, const TlasInst* inst, const float* fwd, uint32_t n, float*, cudaStream_t st) {
    reads(st, inst, sizeof(TlasInst) * n, "the instance records");
    reads(st, fwd, sizeof(float) * 12 * n, "the instance transforms");
    return RQ_OK;
}
int rq_launch_trace_tlas(rq_ctx*, const rq_tlas*, const rq_ray*, uint32_t, uint32_t, uint32_t, rq_hit*, cudaStream_t) {
    return RQ_OK;
}
extern "C" {
int rq_build(rq_ctx*, const float*, uint32_t, uint32_t, const uint32_t*, uint32_t, uint32_t, uint32_t, rq_bvh** out,
             rq_stream) {
    *out = new rq_bvh();
    (*out)->h_counts[2] = 3;
    return RQ_OK;
}
int rq_bvh_destroy(rq_bvh* b) {
    delete b;
    return RQ_OK;
}
int rq_bvh_info_get(rq_bvh*, rq_bvh_info* info) {
    info->depth4 = 2;
    return RQ_OK;
}
}

int main() {
    rq_ctx ctx;
    ctx.num_sms = 148;
    const cudaStream_t side = reinterpret_cast<cudaStream_t>(uintptr_t(0x1000));  // a non-blocking stream
    const float pos[9] = {};
    const uint32_t idx[3] = {};

    const rq_mesh_desc meshes[2] = {{0, 3, 0, 1}, {3, 3, 1, 1}};
    rq_batch* batch = nullptr;
    if (rq_batch_create(&ctx, meshes, 2, 4, &batch) != RQ_OK) return 2;
    if (rq_batch_build(&ctx, batch, pos, 12, idx, side) != RQ_OK) return 2;
    rq_batch_destroy(batch);

    rq_bvh blas;
    blas.has4 = blas.built = true;
    rq_instance inst[2] = {};
    for (rq_instance& i : inst) {
        i.transform[0] = i.transform[5] = i.transform[10] = 1.0f;
        i.mask = 0xff;
        i.blas = &blas;
    }
    rq_tlas* tlas = nullptr;
    if (rq_tlas_build(&ctx, inst, 2, &tlas, side) != RQ_OK) return 2;
    rq_tlas_destroy(tlas);
    return failures ? 1 : 0;
}
