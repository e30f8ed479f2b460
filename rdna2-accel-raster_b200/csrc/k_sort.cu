// k_sort.cu — stable LSD radix sorts of (key, value) pairs, 8 bits a pass, in
// two forms chosen by length (rq_launch_sort), and a single-pass decoupled
// look-back exclusive scan over uint32.
//  - Up to kLookBackMax keys, the onesweep form (Adinets & Merrill 2022): one
//    upfront histogram for every digit position, then one kernel per pass
//    that ranks a tile, resolves its digit offsets by look-back over the
//    preceding tiles, and scatters through shared memory.  A batch of sorts
//    shares the launches.
//  - More keys: the tiles' digit counts, their prefix over the tiles, and a
//    scatter, three kernels a pass with no waiting between tiles.
// Measured (all passes, kernel times): 4,096 keys 81 -> 39 us, 99,458 keys
// 86 -> 48 us (tiles of 1,024 keys in place of 4,608); 2.5M keys 227 ->
// 131 us, 8.3M keys 577 -> 267 us (counted in place of look-back).  The line
// lies where the look-back tiles fill one wave: beyond it every tile waits on
// a chain of tiles that started with it, and the counted form's second read
// of the keys costs less than that.
//
// Look-back tiles are claimed in launch order through an atomic ticket, so a
// tile only ever waits on tiles whose blocks are already running; every wait
// is bounded (RQ_SPIN_LIMIT) and records RQ_DERR_* on the context's error word.
#include <algorithm>

#include "rq_device.cuh"
#include "rq_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 4;                       // keys per thread of a look-back tile
constexpr int kTile = kThreads * kItems;
constexpr uint32_t kLookBackMax = kTile * 148 * 4;  // keys sorted by look-back: one wave of tiles
constexpr int kBigItems = 16;                   // keys per thread of a counted tile
constexpr uint32_t kBigTile = kThreads * kBigItems;
static_assert(kBigTile == RQ_SORT_TILE, "a counted tile");
constexpr int kRadix = 256;
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;
constexpr uint32_t kSpinLimit = 1u << 21;

__global__ void __launch_bounds__(kThreads) k_hist(const uint32_t* __restrict__ keys, uint32_t n, size_t stride,
                                                   uint32_t passes, uint32_t* __restrict__ hist) {
    keys += blockIdx.y * stride;
    hist += blockIdx.y * 4u * kRadix;
    // one private histogram per warp pair to thin out shared-atomic collisions
    __shared__ uint32_t sh[4][4][kRadix];
    uint32_t* flat = &sh[0][0][0];
    for (int i = threadIdx.x; i < 4 * 4 * kRadix; i += kThreads) flat[i] = 0;
    __syncthreads();
    const int copy = (threadIdx.x >> 6) & 3;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        uint32_t k = keys[i];
        for (uint32_t p = 0; p < passes; ++p) atomicAdd(&sh[copy][p][(k >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * kRadix; i += kThreads) {
        int p = i >> 8, d = i & 255;
        uint32_t v = sh[0][p][d] + sh[1][p][d] + sh[2][p][d] + sh[3][p][d];
        if (v) atomicAdd(&hist[i], v);
    }
}

// Block-wide exclusive scan of one value per thread (256 threads).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kWarps) s_warp[lane] = w;  // inclusive warp prefix
    }
    __syncthreads();
    uint32_t warp_prefix = warp ? s_warp[warp - 1] : 0u;
    if (total) *total = s_warp[kWarps - 1];
    uint32_t r = warp_prefix + x - v;
    __syncthreads();
    return r;
}

// Exclusive scan of each pass's 256 bins, in place.
__global__ void __launch_bounds__(kThreads) k_hist_scan(uint32_t* hist) {
    __shared__ uint32_t s_warp[kWarps];
    uint32_t* h = hist + (blockIdx.y * 4u + blockIdx.x) * kRadix;
    uint32_t v = h[threadIdx.x];
    uint32_t ex = block_exclusive_scan(v, s_warp, nullptr);
    h[threadIdx.x] = ex;
}

// Lanes of `act` (all that call this) whose 8-bit digit equals this lane's:
// eight votes.  (__match_any_sync took longer: the 8.3M-key pass 141 against
// 130 us, both in the look-back form.)
__device__ __forceinline__ uint32_t digit_peers(uint32_t act, uint32_t d) {
    uint32_t peers = act;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(act, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// One 8-bit pass over a tile of kTile keys; blockIdx.y is the sort of a batch
// (its arrays `stride` keys further on).  The keys and values go to shared
// memory in digit order before the look-back, which the tile's own counts
// allow, so a tile that waits holds little.  A short launch is bound by the
// steps one block takes one after another: 4,096 keys took 17 us per pass in
// one tile of 4,608 (18 ranking steps per warp), 8.6 us in four of 1,024.
__global__ void __launch_bounds__(kThreads, 4) k_onesweep(const uint32_t* __restrict__ keys_in,
                                                       const uint32_t* __restrict__ vals_in,
                                                       uint32_t* __restrict__ keys_out,
                                                       uint32_t* __restrict__ vals_out, uint32_t n, size_t stride,
                                                       uint32_t shift, const uint32_t* __restrict__ pass_base,
                                                       uint32_t* status, uint32_t* tile_ctr, uint32_t* err) {
    constexpr int ITEMS = kItems;
    constexpr int kWindow = 16;
    __shared__ uint32_t s_cnt[kWarps][kRadix];
    __shared__ uint32_t s_keys[kTile];
    __shared__ uint32_t s_vals[kTile];
    __shared__ uint32_t s_dig_off[kRadix];
    __shared__ uint32_t s_glob[kRadix];
    __shared__ uint32_t s_warp[kWarps];
    __shared__ uint32_t s_tile;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr + blockIdx.y, 1u);
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t tile_base = tile * kTile;
    keys_in += blockIdx.y * stride;
    vals_in += blockIdx.y * stride;
    keys_out += blockIdx.y * stride;
    vals_out += blockIdx.y * stride;
    pass_base += blockIdx.y * 4u * kRadix;
    status += size_t(blockIdx.y) * gridDim.x * kRadix;

    const uint32_t d = threadIdx.x;  // this thread's digit
    uint32_t total = 0;              // its keys in the tile
    {
        uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            uint32_t idx = tile_base + warp * (32 * ITEMS) + j * 32 + lane;
            bool valid = idx < n;
            key[j] = valid ? keys_in[idx] : 0u;
            val[j] = valid ? vals_in[idx] : 0u;
        }
        // Rank within the warp, item by item in tile order: peers with the same
        // digit get consecutive ranks in lane order (stable).
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            uint32_t idx = tile_base + warp * (32 * ITEMS) + j * 32 + lane;
            bool valid = idx < n;
            uint32_t act = __ballot_sync(0xffffffffu, valid);
            rank[j] = 0;
            if (valid) {
                uint32_t d = (key[j] >> shift) & 255u;
                uint32_t peers = digit_peers(act, d);
                int leader = __ffs(peers) - 1;
                uint32_t below = __popc(peers & ((1u << lane) - 1u));
                uint32_t base = 0;
                if (lane == leader) {
                    base = s_cnt[warp][d];
                    s_cnt[warp][d] = base + __popc(peers);
                }
                base = __shfl_sync(peers, base, leader);
                rank[j] = base + below;
            }
            __syncwarp();
        }
        __syncthreads();
        // warp-exclusive offsets and tile total
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            uint32_t c = s_cnt[w][d];
            s_cnt[w][d] = total;
            total += c;
        }
        // publish the tile's count early so successors can proceed
        if (tile != 0) rq::st_release(&status[size_t(tile) * kRadix + d], kFlagAgg | total);
        s_dig_off[d] = block_exclusive_scan(total, s_warp, nullptr);
        __syncthreads();
        // into shared memory in digit order
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            uint32_t idx = tile_base + warp * (32 * ITEMS) + j * 32 + lane;
            if (idx < n) {
                uint32_t dj = (key[j] >> shift) & 255u;
                uint32_t pos = s_dig_off[dj] + s_cnt[warp][dj] + rank[j];
                s_keys[pos] = key[j];
                s_vals[pos] = val[j];
            }
        }
    }
    // decoupled look-back for this digit
    uint32_t glob;
    if (tile == 0) {
        glob = pass_base[d];
        rq::st_release(&status[d], kFlagPrefix | (glob + total));
    } else {
        // The statuses of the kWindow nearest unvisited predecessors are read
        // at once (relaxed loads: each count shares its word with its flag,
        // and nothing else the predecessor wrote is read), then walked nearest
        // first until an inclusive prefix; a predecessor not yet published
        // ends the window and is read again.
        uint32_t acc = 0, spins = 0;
        int t = int(tile) - 1;
        for (;;) {
            uint32_t st[kWindow];
#pragma unroll
            for (int q = 0; q < kWindow; ++q)
                st[q] = t - q >= 0 ? rq::ld_relaxed(&status[size_t(t - q) * kRadix + d]) : 0u;
            int used = 0;
            bool done = false;
#pragma unroll
            for (int q = 0; q < kWindow; ++q) {
                if (done || used < q) continue;  // stopped earlier in this window
                const uint32_t flag = st[q] & ~kValueMask;
                if (flag == 0u) continue;        // not yet published: read again from here
                acc += st[q] & kValueMask;
                used = q + 1;
                done = flag == kFlagPrefix;
            }
            if (done) break;
            if (used == 0 && ++spins > kSpinLimit) {
                rq::set_err(err, RQ_DERR_SORT_LOOKBACK);
                break;
            }
            t -= used;
        }
        glob = acc;
        rq::st_release(&status[size_t(tile) * kRadix + d], kFlagPrefix | (acc + total));
    }
    s_glob[d] = glob - s_dig_off[d];
    __syncthreads();
    const uint32_t tile_n = n - tile_base < uint32_t(kTile) ? n - tile_base : uint32_t(kTile);
    for (uint32_t i = threadIdx.x; i < tile_n; i += kThreads) {
        uint32_t k = s_keys[i];
        uint32_t g = s_glob[(k >> shift) & 255u] + i;
        keys_out[g] = k;
        vals_out[g] = s_vals[i];
    }
}

// ------------------------------------------------------------ counted form
// More keys than one wave of look-back tiles holds: per pass the tiles' digit
// counts, their prefix over the tiles, and a scatter that waits for nothing.
// A look-back over 8.3M keys (1,807 tiles of 4,608) took 130 us per pass: 239
// warp instructions per 32 keys, a third of them walking status windows, and
// a chain of L2 round trips.
// The keys [base, base + count) of tile blockIdx.x: the next kBigTile of one
// sort of n keys, or tiles[blockIdx.x] of a sort of segments.
__device__ __forceinline__ void tile_range(const rq_sort_tile* tiles, uint32_t n, uint32_t& base, uint32_t& count,
                                           uint32_t& seg) {
    if (tiles) {
        const rq_sort_tile t = tiles[blockIdx.x];
        base = t.first;
        count = t.count;
        seg = t.seg_first;
    } else {
        base = blockIdx.x * kBigTile;
        count = min(kBigTile, n - base);
        seg = 0;
    }
}

__global__ void __launch_bounds__(kThreads) k_tile_count(const uint32_t* __restrict__ keys, uint32_t n, uint32_t shift,
                                                         const rq_sort_tile* __restrict__ tiles,
                                                         uint32_t* __restrict__ counts) {
    __shared__ uint32_t sh[4][kRadix];
    uint32_t* mine = sh[(threadIdx.x >> 6) & 3];
    for (int i = threadIdx.x; i < 4 * kRadix; i += kThreads) (&sh[0][0])[i] = 0;
    __syncthreads();
    uint32_t base, count, seg;
    tile_range(tiles, n, base, count, seg);
    if (count == kBigTile && base % 4 == 0) {
        const uint4* k4 = reinterpret_cast<const uint4*>(keys + base);
#pragma unroll
        for (int j = 0; j < kBigItems / 4; ++j) {
            const uint4 k = k4[j * kThreads + threadIdx.x];
            atomicAdd(mine + ((k.x >> shift) & 255u), 1u);
            atomicAdd(mine + ((k.y >> shift) & 255u), 1u);
            atomicAdd(mine + ((k.z >> shift) & 255u), 1u);
            atomicAdd(mine + ((k.w >> shift) & 255u), 1u);
        }
    } else {
        for (uint32_t i = threadIdx.x; i < count; i += kThreads) atomicAdd(mine + ((keys[base + i] >> shift) & 255u), 1u);
    }
    __syncthreads();
    const uint32_t d = threadIdx.x;
    counts[size_t(blockIdx.x) * kRadix + d] = sh[0][d] + sh[1][d] + sh[2][d] + sh[3][d];
}

// A segment's tiles by one block (thread = digit): each digit's first place in
// the segment plus its count in the tiles before, in place of the counts.
__global__ void __launch_bounds__(kThreads) k_segment_prefix(uint32_t* counts, const uint32_t* __restrict__ seg_tiles) {
    __shared__ uint32_t s_warp[kWarps];
    const uint32_t t0 = seg_tiles[blockIdx.x], t1 = seg_tiles[blockIdx.x + 1], d = threadIdx.x;
    uint32_t total = 0;
#pragma unroll 8
    for (uint32_t t = t0; t < t1; ++t) total += counts[size_t(t) * kRadix + d];
    uint32_t acc = block_exclusive_scan(total, s_warp, nullptr);
#pragma unroll 8
    for (uint32_t t = t0; t < t1; ++t) {
        const uint32_t c = counts[size_t(t) * kRadix + d];
        counts[size_t(t) * kRadix + d] = acc;
        acc += c;
    }
}

// Exclusive prefix of every digit's counts over the tiles, in place, and the
// digits' totals.  A block takes 8 digits (a 32-byte sector of each row), its
// threads a run of tiles each.
constexpr int kPrefixThreads = 1024;
constexpr uint32_t kPrefixDigits = 8, kPrefixRuns = kPrefixThreads / kPrefixDigits;
__global__ void __launch_bounds__(kPrefixThreads) k_tile_prefix(uint32_t* counts, uint32_t tiles,
                                                                uint32_t* __restrict__ totals) {
    __shared__ uint32_t s_sum[kPrefixRuns][kPrefixDigits + 1];
    const uint32_t dl = threadIdx.x % kPrefixDigits, run = threadIdx.x / kPrefixDigits;
    const uint32_t d = blockIdx.x * kPrefixDigits + dl;
    const uint32_t per = (tiles + kPrefixRuns - 1) / kPrefixRuns;
    const uint32_t t0 = min(run * per, tiles), t1 = min(t0 + per, tiles);
    uint32_t sum = 0;
#pragma unroll 8
    for (uint32_t t = t0; t < t1; ++t) sum += counts[size_t(t) * kRadix + d];
    s_sum[run][dl] = sum;
    __syncthreads();
    // warp w < 8: digit w's runs, 4 per lane
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (warp < kPrefixDigits) {
        constexpr uint32_t kPer = kPrefixRuns / 32;
        uint32_t v[kPer], s = 0;
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            v[i] = s_sum[lane * kPer + i][warp];
            s += v[i];
        }
        uint32_t x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (int(lane) >= o) x += y;
        }
        if (lane == 31) totals[blockIdx.x * kPrefixDigits + warp] = x;
        uint32_t ex = x - s;
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            s_sum[lane * kPer + i][warp] = ex;
            ex += v[i];
        }
    }
    __syncthreads();
    uint32_t acc = s_sum[run][dl];
#pragma unroll 8
    for (uint32_t t = t0; t < t1; ++t) {
        const uint32_t c = counts[size_t(t) * kRadix + d];
        counts[size_t(t) * kRadix + d] = acc;
        acc += c;
    }
}

// (At 64 registers, 4 blocks per SM, it spills 156 bytes.  8, 12 and 16 keys per
// thread and 3 and 4 blocks took 184 to 198 us for the four passes over 8.3M
// keys, near what DRAM moves, so the spills stay.)
// Stable scatter of one tile: ranks within the warp (the lanes of a digit read
// its count together, the first one adds them), then digit order in shared
// memory, then runs to their places.
template <bool FULL>
__device__ __forceinline__ void scatter_tile(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                             uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                             uint32_t base, uint32_t n, uint32_t seg, uint32_t shift,
                                             const uint32_t* __restrict__ prefix, const uint32_t* __restrict__ totals,
                                             uint32_t (*s_cnt)[kRadix], uint32_t* s_keys, uint32_t* s_vals,
                                             uint32_t* s_glob, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t first = base + warp * (32 * kBigItems) + lane;  // (n: the tile's end)
    uint32_t key[kBigItems], val[kBigItems], rank[kBigItems];
#pragma unroll
    for (int j = 0; j < kBigItems; ++j) {
        const bool valid = FULL || first + j * 32 < n;
        key[j] = valid ? keys_in[first + j * 32] : 0u;
        val[j] = valid ? vals_in[first + j * 32] : 0u;
    }
    const uint32_t d = threadIdx.x;
    const uint32_t tot = totals ? totals[d] : 0u, pre = prefix[d];
    uint32_t* cnt = s_cnt[warp];
#pragma unroll
    for (int j = 0; j < kBigItems; ++j) {
        const bool valid = FULL || first + j * 32 < n;
        const uint32_t act = FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, valid);
        rank[j] = 0;
        if (!FULL && !act) break;
        if (valid) {
            const uint32_t dj = (key[j] >> shift) & 255u;
            const uint32_t peers = digit_peers(act, dj);
            const uint32_t below = __popc(peers & lt);
            const uint32_t c = cnt[dj];
            __syncwarp(act);
            if (below == 0) cnt[dj] = c + __popc(peers);
            rank[j] = c + below;
        }
        __syncwarp();
    }
    __syncthreads();  // every warp's counts
    // the digits' first places over all keys, and in the tile
    // (a segment's prefix has its digits' places in it)
    const uint32_t digit_base = totals ? block_exclusive_scan(tot, s_warp, nullptr) : seg;
    uint32_t mine = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mine += s_cnt[w][d];
    uint32_t run = block_exclusive_scan(mine, s_warp, nullptr);
    s_glob[d] = digit_base + pre - run;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = s_cnt[w][d];
        s_cnt[w][d] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kBigItems; ++j)
        if (FULL || first + j * 32 < n) {
            const uint32_t at = cnt[(key[j] >> shift) & 255u] + rank[j];
            s_keys[at] = key[j];
            s_vals[at] = val[j];
        }
    __syncthreads();
    const uint32_t count = FULL ? kBigTile : n - base;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < count; i += kThreads) {
        const uint32_t k = s_keys[i], g = s_glob[(k >> shift) & 255u] + i;
        keys_out[g] = k;
        vals_out[g] = s_vals[i];
    }
}

__global__ void __launch_bounds__(kThreads, 4) k_tile_scatter(const uint32_t* __restrict__ keys_in,
                                                              const uint32_t* __restrict__ vals_in,
                                                              uint32_t* __restrict__ keys_out,
                                                              uint32_t* __restrict__ vals_out, uint32_t n,
                                                              uint32_t shift, const rq_sort_tile* __restrict__ tiles,
                                                              const uint32_t* __restrict__ prefix,
                                                              const uint32_t* __restrict__ totals) {
    __shared__ uint32_t s_cnt[kWarps][kRadix];
    __shared__ uint32_t s_keys[kBigTile];
    __shared__ uint32_t s_vals[kBigTile];
    __shared__ uint32_t s_glob[kRadix];
    __shared__ uint32_t s_warp[kWarps];
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    prefix += size_t(blockIdx.x) * kRadix;
    uint32_t base, count, seg;
    tile_range(tiles, n, base, count, seg);
    if (count == kBigTile)
        scatter_tile<true>(keys_in, vals_in, keys_out, vals_out, base, base + count, seg, shift, prefix, totals, s_cnt,
                           s_keys, s_vals, s_glob, s_warp);
    else
        scatter_tile<false>(keys_in, vals_in, keys_out, vals_out, base, base + count, seg, shift, prefix, totals, s_cnt,
                            s_keys, s_vals, s_glob, s_warp);
}

// ------------------------------------------------------------------ scan
// Items per thread: the prefixes travel 32 tiles at a time, so long arrays take
// larger tiles (8.3M emission counts: 52 us at 8 items, 34 at 32; 4.7M 33 and
// 25; 2.5M 18.5 and 19.6, so the line lies between).
constexpr int kScanItems = 8, kScanItemsLong = 32;
constexpr uint32_t kScanLong = 1u << 22;
constexpr int kScanTile = kThreads * kScanItems;

__device__ __forceinline__ void scan_words(const uint32_t* in, uint32_t* v) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(in)), b = __ldg(reinterpret_cast<const uint4*>(in) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void scan_words(const uint16_t* in, uint32_t* v) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(in));
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (w[i >> 1] >> (16 * (i & 1))) & 255u;
}
__device__ __forceinline__ uint32_t scan_word(const uint32_t* in) { return *in; }
__device__ __forceinline__ uint32_t scan_word(const uint16_t* in) { return *in & 255u; }

// In: 32-bit words, or the low bytes of 16-bit ones (16-byte aligned).
template <class In, int ITEMS>
__global__ void __launch_bounds__(kThreads) k_scan(const In* __restrict__ in, uint32_t* __restrict__ out,
                                                   uint32_t n, uint32_t* status, uint32_t* tile_ctr, uint32_t* err) {
    __shared__ uint32_t s_warp[kWarps];
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * (kThreads * ITEMS) + threadIdx.x * ITEMS;
    uint32_t v[ITEMS];
    uint32_t sum = 0;
    const bool full = base + ITEMS <= n;
    if (full) {
#pragma unroll
        for (int i = 0; i < ITEMS; i += 8) scan_words(in + base + i, v + i);
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) v[i] = base + i < n ? scan_word(in + base + i) : 0u;
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) sum += v[i];
    uint32_t total;
    uint32_t ex = block_exclusive_scan(sum, s_warp, &total);
    if (threadIdx.x < 32) {
        // warp-wide decoupled look-back: 32 predecessors per step; the
        // nearest one with its inclusive prefix ends the walk
        const uint32_t lane = threadIdx.x;
        if (tile == 0) {
            if (lane == 0) {
                rq::st_release(&status[0], kFlagPrefix | total);
                s_prefix = 0;
            }
        } else {
            if (lane == 0) rq::st_release(&status[tile], kFlagAgg | total);
            uint32_t acc = 0, spins = 0;
            for (int t0 = int(tile) - 1;; t0 -= 32) {
                const int t = t0 - int(lane);
                uint32_t st = kFlagPrefix;  // before tile 0: an inclusive prefix of 0
                if (t >= 0) {
                    for (;;) {
                        st = rq::ld_acquire(&status[t]);
                        if (st & ~kValueMask) break;
                        if (++spins > kSpinLimit) {
                            rq::set_err(err, RQ_DERR_SCAN_LOOKBACK);
                            st = kFlagPrefix;
                            break;
                        }
                    }
                }
                const uint32_t pm = __ballot_sync(0xffffffffu, (st & ~kValueMask) == kFlagPrefix);
                uint32_t val = st & kValueMask;
                if (pm && int(lane) > __ffs(pm) - 1) val = 0u;
                acc += __reduce_add_sync(0xffffffffu, val);
                if (pm) break;
            }
            if (lane == 0) {
                rq::st_release(&status[tile], kFlagPrefix | (acc + total));
                s_prefix = acc;
            }
        }
    }
    __syncthreads();
    uint32_t run = s_prefix + ex;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t x = v[i];
        v[i] = run;
        run += x;
    }
    if (full) {
        uint4* o = reinterpret_cast<uint4*>(out + base);
#pragma unroll
        for (int i = 0; i < ITEMS; i += 4) o[i / 4] = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (base + i < n) out[base + i] = v[i];
    }
}

}  // namespace

uint32_t rq_scan_tiles(uint32_t n) { return (n + kScanTile - 1) / kScanTile; }

namespace {
uint32_t tiles_of(uint32_t n, uint32_t tile) { return (n + tile - 1) / tile; }
}  // namespace

// (never fewer for more keys, whichever form sorts them)
size_t rq_sort_words(uint32_t n, uint32_t batch) {
    const size_t look_back = size_t(batch) * kRadix * 4 * (1 + tiles_of(std::min(n, kLookBackMax), kTile)) + 4 * batch;
    const size_t counted = n > kLookBackMax ? size_t(kRadix) * (tiles_of(n, kBigTile) + 1) : 0;
    return std::max(look_back, counted);
}

int rq_launch_sort(rq_ctx* ctx, const SortIO& io, uint32_t n, uint32_t bits, uint32_t batch, cudaStream_t st,
                   int* result_buf) {
    const uint32_t passes = (bits + 7) / 8;
    *result_buf = int(passes & 1);
    if (n > kLookBackMax) {
        const uint32_t tiles = tiles_of(n, kBigTile);
        uint32_t *counts = io.words, *totals = counts + size_t(tiles) * kRadix;
        for (uint32_t y = 0; y < batch; ++y)
            for (uint32_t p = 0; p < passes; ++p) {
                const int a = int(p & 1), b = 1 - a;
                const size_t o = y * io.stride;
                k_tile_count<<<tiles, kThreads, 0, st>>>(io.keys[a] + o, n, 8 * p, nullptr, counts);
                k_tile_prefix<<<kRadix / kPrefixDigits, kPrefixThreads, 0, st>>>(counts, tiles, totals);
                k_tile_scatter<<<tiles, kThreads, 0, st>>>(io.keys[a] + o, io.vals[a] + o, io.keys[b] + o,
                                                           io.vals[b] + o, n, 8 * p, nullptr, counts, totals);
            }
        return rq_cuda_status(ctx, cudaGetLastError(), "radix sort launch");
    }
    const uint32_t tiles = tiles_of(n, kTile);
    // one block of words, zeroed at once: the histograms, the tiles' statuses
    // of every pass, the tile tickets
    uint32_t* hist = io.words;
    uint32_t* status = hist + size_t(batch) * 4 * kRadix;
    uint32_t* ticket = status + size_t(batch) * passes * tiles * kRadix;
    cudaError_t e = cudaMemsetAsync(
        io.words, 0, sizeof(uint32_t) * (size_t(batch) * (4 * kRadix + size_t(passes) * tiles * kRadix) + passes * batch),
        st);
    if (e != cudaSuccess) return rq_cuda_status(ctx, e, "radix sort scratch");
    const uint32_t hist_blocks = std::min((n + 4 * kThreads - 1) / (4 * kThreads), uint32_t(2 * ctx->num_sms));
    k_hist<<<dim3(hist_blocks, batch), kThreads, 0, st>>>(io.keys[0], n, io.stride, passes, hist);
    k_hist_scan<<<dim3(passes, batch), kThreads, 0, st>>>(hist);
    for (uint32_t p = 0; p < passes; ++p) {
        const int a = int(p & 1), b = 1 - a;
        k_onesweep<<<dim3(tiles, batch), kThreads, 0, st>>>(io.keys[a], io.vals[a], io.keys[b], io.vals[b], n,
                                                            io.stride, 8 * p, hist + kRadix * p,
                                                            status + size_t(p) * batch * tiles * kRadix,
                                                            ticket + p * batch, ctx->d_err);
    }
    return rq_cuda_status(ctx, cudaGetLastError(), "radix sort launch");
}

int rq_launch_sort_tiles(rq_ctx* ctx, const SortIO& io, const rq_sort_tile* tiles, uint32_t ntiles,
                         const uint32_t* seg_tiles, uint32_t nsegs, uint32_t bits, cudaStream_t st, int* result_buf) {
    const uint32_t passes = (bits + 7) / 8;
    for (uint32_t p = 0; p < passes; ++p) {
        const int a = int(p & 1), b = 1 - a;
        k_tile_count<<<ntiles, kThreads, 0, st>>>(io.keys[a], 0, 8 * p, tiles, io.words);
        k_segment_prefix<<<nsegs, kThreads, 0, st>>>(io.words, seg_tiles);
        k_tile_scatter<<<ntiles, kThreads, 0, st>>>(io.keys[a], io.vals[a], io.keys[b], io.vals[b], 0, 8 * p, tiles,
                                                    io.words, nullptr);
    }
    *result_buf = int(passes & 1);
    return rq_cuda_status(ctx, cudaGetLastError(), "segment sort launch");
}

template <class In>
static void launch_scan(rq_ctx* ctx, const In* in, uint32_t* out, uint32_t n, uint32_t* status, uint32_t* tile_ctr,
                        cudaStream_t st) {
    const bool lng = n >= kScanLong;
    const uint32_t tile = kThreads * uint32_t(lng ? kScanItemsLong : kScanItems), tiles = (n + tile - 1) / tile;
    cudaMemsetAsync(status, 0, sizeof(uint32_t) * tiles, st);
    auto k = lng ? k_scan<In, kScanItemsLong> : k_scan<In, kScanItems>;
    k<<<tiles, kThreads, 0, st>>>(in, out, n, status, tile_ctr, ctx->d_err);
}
void rq_launch_scan(rq_ctx* ctx, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* status, uint32_t* tile_ctr,
                    cudaStream_t st) {
    launch_scan(ctx, in, out, n, status, tile_ctr, st);
}
void rq_launch_scan(rq_ctx* ctx, const uint16_t* in, uint32_t* out, uint32_t n, uint32_t* status, uint32_t* tile_ctr,
                    cudaStream_t st) {
    launch_scan(ctx, in, out, n, status, tile_ctr, st);
}
