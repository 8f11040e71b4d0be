// radix_sort.cuh — stable LSD radix sort of (u32 key, u32 value) pairs.
//
// One kernel per 8-bit digit pass, after one that counts the digits of every
// pass (k_rs_count, or the kernel that makes the keys: rs_count_key).  A pass
// reads its tile once: it ranks the tile's items among equal digits (a ballot per
// bit of the digit per 32-item round, per-warp counters in shared memory), learns how
// many of each digit the tiles before it hold by decoupled look-back (Merrill
// and Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back",
// 2016; one thread per digit), and writes the items, ordered by digit in shared
// memory first, so that the items of a digit leave in runs.
//
// Bound by the chain of launches for small counts; for large ones by what a
// tile does once (ranking, look-back of 256 digits) at 1.7 tiles per SM for 1M
// pairs.  Against three kernels per pass (tile histograms, a scan of every
// digit's row, a scatter straight from registers), the whole device-resident
// grid of 1,000,003 / 300,000 / 20,000 / 300 photons: 99 -> 81, 68 -> 58, 62 -> 46
// and 54 -> 36 us; the photon pass of config 1 0.330 -> 0.305 ms.  Tiles of 2048 /
// 8192 items kept in registers: 96, 96 us for the first.
//
// Tiles take their numbers from a counter in the order in which they start, so
// the tiles a look-back waits for are running; its polls are bounded all the
// same (RS_POLLS), and a tile that gives up sets RS_GAVE_UP in the scratch, as
// does a block whose number is none of a tile's (launches that share a scratch
// overlap): the result is then to be dropped.
// The element count may live in device memory (n_dev), so the same launches
// serve a count produced on the GPU and can be captured in a CUDA graph; tiles
// at or beyond the count exit at once.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <cuda_runtime.h>

namespace srt {

constexpr int RS_WARPS = 16;
constexpr int RS_THREADS = RS_WARPS * 32;
constexpr int RS_IPT = 8;                        // items per thread per tile
constexpr int RS_TILE = RS_THREADS * RS_IPT;     // 4096 items
constexpr int RS_PASSES = 4;                     // most digit passes of a sort
constexpr uint32_t RS_POLLS = 1u << 16;

// Scratch words: digit counts of each pass, a tile counter per pass, a flag,
// then two arrays of a status word per tile and digit (a pass clears its part of
// the next pass's).  A status word: 0 (nothing yet), RS_SUM | items of the digit
// in this tile, or RS_PREFIX | items in this tile and all before it.
constexpr uint32_t RS_HIST = 0, RS_TICKET = RS_PASSES * 256, RS_GAVE_UP = RS_TICKET + RS_PASSES,
                   RS_HEAD = RS_GAVE_UP + 4;
constexpr uint32_t RS_SUM = 1u << 30, RS_PREFIX = 2u << 30, RS_COUNT = RS_SUM - 1u;

constexpr uint32_t rs_tiles(uint32_t n) { return (uint32_t)(((uint64_t)n + RS_TILE - 1) / RS_TILE); }
constexpr size_t radix_scratch_words(uint32_t max_n) {
    return RS_HEAD + 2ull * 256 * (rs_tiles(max_n) ? rs_tiles(max_n) : 1);
}

__device__ __forceinline__ uint32_t rs_count(const uint32_t* n_dev, uint32_t n_host) {
    return n_dev ? *n_dev : n_host;
}

// Clears the scratch's head (before the digits are counted) or the first status
// array (before the first pass), by all threads of a launch.
__device__ __forceinline__ void rs_clear(uint32_t* words, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) words[i] = 0u;
}
__device__ __forceinline__ void rs_clear_status(uint32_t* scratch, uint32_t n) {
    rs_clear(scratch + RS_HEAD, 256u * ((n + RS_TILE - 1u) / RS_TILE));
}
// A key's digits into the block's counts h[passes * 256] (shared memory,
// cleared before; rs_flush_counts adds them to the scratch's).
__device__ __forceinline__ void rs_count_key(uint32_t* h, uint32_t key, int begin_bit, int passes) {
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p * 256 + ((key >> (begin_bit + 8 * p)) & 0xFFu)], 1u);
}
__device__ __forceinline__ void rs_flush_counts(const uint32_t* h, uint32_t* scratch, int passes) {
    for (int i = (int)threadIdx.x; i < passes * 256; i += (int)blockDim.x)
        if (h[i] != 0u) atomicAdd(&scratch[RS_HIST + i], h[i]);
}

static __global__ void __launch_bounds__(RS_THREADS) k_rs_count(const uint32_t* __restrict__ keys, const uint32_t* n_dev,
                                                          uint32_t n_host, int begin_bit, int passes,
                                                          uint32_t* __restrict__ scratch) {
    __shared__ uint32_t h[RS_PASSES * 256];
    for (int i = threadIdx.x; i < RS_PASSES * 256; i += RS_THREADS) h[i] = 0u;
    __syncthreads();
    const uint32_t n = rs_count(n_dev, n_host);
    rs_clear_status(scratch, n);
    for (uint32_t i = blockIdx.x * RS_THREADS + threadIdx.x; i < n; i += gridDim.x * RS_THREADS)
        rs_count_key(h, keys[i], begin_bit, passes);
    __syncthreads();
    rs_flush_counts(h, scratch, passes);
}

// Exclusive prefix sum of one value per thread over a block of RS_THREADS.
__device__ __forceinline__ uint32_t rs_block_exclusive(uint32_t v, uint32_t* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t add = 0;
    for (int w = 0; w < warp; ++w) add += warp_sums[w];
    __syncthreads();
    return add + x - v;
}

// Items of this thread's status column before tile `tile`: look-back over the
// words status[t * stride], t < tile, RS_WINDOW of them loaded at once (a load
// takes an L2 round trip, and the prefix is many tiles away when all start
// together; loads beyond it are wasted, and 256 digits of 245 tiles of them are
// what a pass of 1M pairs waits for).  Windows of 2 / 3 / 4 / 5 / 6 / 8 / 16 / 32:
// the device-resident grid of 1,000,003 photons 87.3 / 81.2 / 81.3 / 81.4 / 81.6 /
// 86.5 / 89.0 / 97.2 us, of 300,000 62.2 / 58.3 / 58.5 / 57.9 / 58.0 / 58.8 / 61.4 /
// 61.5, of 2^20 with 24-bit keys 132 / 129 / 129 / 128 / 130 / 132 / 139 / 147.
constexpr uint32_t RS_WINDOW = 5;
__device__ __forceinline__ uint32_t rs_look_back(const uint32_t* status, uint32_t stride, uint32_t tile,
                                                 uint32_t* gave_up) {
    uint32_t before = 0u;
    for (uint32_t t = tile; t > 0u;) {
        uint32_t s[RS_WINDOW];
#pragma unroll
        for (uint32_t j = 0; j < RS_WINDOW; ++j)
            s[j] = j < t ? *(const volatile uint32_t*)(status + (size_t)(t - 1u - j) * stride) : RS_PREFIX;
        bool done = false;
#pragma unroll
        for (uint32_t j = 0; j < RS_WINDOW; ++j) {
            if (done) continue;
            uint32_t w = s[j];
            for (uint32_t polls = 0; w == 0u && polls < RS_POLLS; ++polls)
                w = *(const volatile uint32_t*)(status + (size_t)(t - 1u - j) * stride);
            if (w == 0u) {
                atomicOr(gave_up, 1u);
                w = RS_PREFIX;
            }
            before += w & RS_COUNT;
            done = (w & RS_PREFIX) != 0u;
        }
        if (done) break;
        t -= RS_WINDOW;
    }
    return before;
}

// The loops over a thread's items stay loops: a tile runs its code once, and
// unrolled (30 KB of it) a block waited for instructions (a single tile of 8192
// items took 15 us).  So the items live in shared memory, not in registers.
static __global__ void __launch_bounds__(RS_THREADS) k_rs_pass(const uint32_t* __restrict__ keys_in,
                                                         const uint32_t* __restrict__ vals_in,
                                                         uint32_t* __restrict__ keys_out,
                                                         uint32_t* __restrict__ vals_out, const uint32_t* n_dev,
                                                         uint32_t n_host, int shift, int pass, uint32_t max_tiles,
                                                         uint32_t* __restrict__ scratch) {
    __shared__ uint32_t keys[RS_TILE];
    __shared__ uint8_t rank[RS_TILE];            // among the warp's 256 items
    __shared__ uint16_t from[RS_TILE];           // the item at each place of the digit order
    __shared__ uint16_t cnt[RS_WARPS][256];
    __shared__ uint32_t digit_base[256], warp_sums[RS_WARPS], ticket;
    const uint32_t n = rs_count(n_dev, n_host);
    const uint32_t tiles = (n + RS_TILE - 1u) / RS_TILE;
    if (blockIdx.x >= tiles) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, lt = (1u << lane) - 1u;
    if (tid == 0) ticket = atomicAdd(&scratch[RS_TICKET + pass], 1u);
    for (uint32_t d = tid; d < RS_WARPS * 128u; d += RS_THREADS) reinterpret_cast<uint32_t*>(&cnt[0][0])[d] = 0u;
    __syncthreads();
    const uint32_t tile = ticket;
    if (tile >= tiles) {  // another launch drew from the same counter (calls that share a scratch overlap)
        if (tid == 0) atomicOr(&scratch[RS_GAVE_UP], 1u);
        return;
    }
    const uint32_t tile_base = tile * (uint32_t)RS_TILE, items = min((uint32_t)RS_TILE, n - tile_base);
    // threads 0 .. 255: one digit each
    const bool digit = tid < 256u;
    uint32_t* status = scratch + RS_HEAD + ((size_t)(pass & 1) * max_tiles + tile) * 256;
    uint32_t total = 0u;  // items of the digit in the whole input
    if (digit) {
        scratch[RS_HEAD + ((size_t)((pass + 1) & 1) * max_tiles + tile) * 256 + tid] = 0u;  // the next pass's
        total = scratch[RS_HIST + pass * 256 + tid];
    }
    {
        uint32_t k[RS_IPT];
#pragma unroll
        for (uint32_t r = 0; r < RS_IPT; ++r) k[r] = r * RS_THREADS + tid < items ? keys_in[tile_base + r * RS_THREADS + tid] : 0u;
#pragma unroll
        for (uint32_t r = 0; r < RS_IPT; ++r) keys[r * RS_THREADS + tid] = k[r];
    }
    __syncthreads();
    // ranks among equal digits of the warp's items, in order
#pragma unroll 1
    for (uint32_t r = 0; r < RS_IPT; ++r) {
        const uint32_t i = warp * 32u * RS_IPT + r * 32u + lane, d = (keys[i] >> shift) & 0xFFu;
        // the lanes with this lane's digit, bit by bit
        uint32_t peers = __ballot_sync(0xFFFFFFFFu, i < items);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? m : ~m;
        }
        const uint32_t before = i < items ? cnt[warp][d] : 0u;
        rank[i] = (uint8_t)(before + __popc(peers & lt));
        __syncwarp();
        if (i < items && (peers & lt) == 0u) cnt[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // the warps' counts become offsets, the tile's count is published, the
    // tiles before it are looked up
    uint32_t run = 0u;
    if (digit) {
#pragma unroll 4
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t c = cnt[w][tid];
            cnt[w][tid] = (uint16_t)run;
            run += c;
        }
        *(volatile uint32_t*)(status + tid) = (tile == 0u ? RS_PREFIX : RS_SUM) | run;
    }
    const uint32_t in_tile = rs_block_exclusive(run, warp_sums);
    const uint32_t smaller = rs_block_exclusive(total, warp_sums);
    if (digit) {
        for (int w = 0; w < RS_WARPS; ++w) cnt[w][tid] = (uint16_t)(cnt[w][tid] + in_tile);
        uint32_t before = 0u;
        if (tile > 0u) {
            before = rs_look_back(status + tid - (size_t)tile * 256, 256u, tile, &scratch[RS_GAVE_UP]);
            *(volatile uint32_t*)(status + tid) = RS_PREFIX | (before + run);
        }
        digit_base[tid] = smaller + before - in_tile;  // of the tile's item at place p of the order: + p
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t r = 0; r < RS_IPT; ++r) {
        const uint32_t i = warp * 32u * RS_IPT + r * 32u + lane;
        if (i < items) from[cnt[warp][(keys[i] >> shift) & 0xFFu] + rank[i]] = (uint16_t)i;
    }
    __syncthreads();
    // out in digit order, so that the items of a digit leave in runs
#pragma unroll 4
    for (uint32_t r = 0; r < RS_IPT; ++r) {
        const uint32_t p = r * RS_THREADS + tid;
        if (p < items) {
            const uint32_t i = from[p], key = keys[i], pos = digit_base[(key >> shift) & 0xFFu] + p;
            if (pos < n) {  // (a look-back that gave up leaves wrong positions)
                keys_out[pos] = key;
                vals_out[pos] = vals_in[tile_base + i];
            }
        }
    }
}

// Host-side fault injection: with SRT_FAULT=sort every sort_pairs counts as one
// whose bounded wait gave up.
inline bool sort_fault() {
    const char* f = std::getenv("SRT_FAULT");
    return f && std::strcmp(f, "sort") == 0;
}

// Digit passes of a sort of bits [begin_bit, end_bit).
constexpr int rs_passes(int begin_bit, int end_bit) { return (end_bit - begin_bit + 7) / 8; }

// The passes of a sort whose digits have been counted and whose first status
// array is clear.  *out_keys / *out_vals receive whichever pair of buffers
// holds the result.  Returns the number of kernels launched.
inline int sort_passes(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t max_n,
                       const uint32_t* n_dev, int begin_bit, int end_bit, uint32_t* scratch, cudaStream_t st,
                       uint32_t** out_keys, uint32_t** out_vals) {
    const uint32_t tiles = rs_tiles(max_n);
    uint32_t *ki = keys, *vi = vals, *ko = keys_alt, *vo = vals_alt;
    const int passes = tiles > 0 ? rs_passes(begin_bit, end_bit) : 0;
    for (int p = 0; p < passes; ++p) {
        k_rs_pass<<<tiles, RS_THREADS, 0, st>>>(ki, vi, ko, vo, n_dev, max_n, begin_bit + 8 * p, p, tiles, scratch);
        std::swap(ki, ko);
        std::swap(vi, vo);
    }
    *out_keys = ki;
    *out_vals = vi;
    return passes;
}

// Sorts bits [begin_bit, end_bit) of (keys, vals), ping-ponging with the
// alternate buffers.  max_n (< 2^30) bounds the count for the launch grid;
// n_dev (optional) holds the actual count.  The caller looks at
// scratch[RS_GAVE_UP] before it uses the result.
inline int sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t max_n,
                      const uint32_t* n_dev, int begin_bit, int end_bit, uint32_t* scratch, cudaStream_t st,
                      uint32_t** out_keys, uint32_t** out_vals) {
    int launches = 0;
    if (max_n > 0) {
        cudaMemsetAsync(scratch, 0, RS_HEAD * sizeof(uint32_t), st);
        k_rs_count<<<std::min(rs_tiles(max_n), 592u), RS_THREADS, 0, st>>>(keys, n_dev, max_n, begin_bit,
                                                                         rs_passes(begin_bit, end_bit), scratch);
        ++launches;
        if (sort_fault()) cudaMemsetAsync(scratch + RS_GAVE_UP, 1, sizeof(uint32_t), st);
    }
    return launches + sort_passes(keys, vals, keys_alt, vals_alt, max_n, n_dev, begin_bit, end_bit, scratch, st, out_keys,
                                  out_vals);
}

}  // namespace srt
