// The cell-list rebuild's device side, shared by the step kernels: a bead's arrival in its new
// cell, and the prefix sum of the cell counts.
#pragma once

#include "pdpd_device.cuh"

namespace pdpd {
namespace {

// A bead's id rides in the spare w of its velocity.
__device__ __forceinline__ float id_word32(uint32_t id) { return __uint_as_float(id); }
__device__ __forceinline__ double id_word64(uint32_t id) { return __longlong_as_double((long long)id); }
__device__ __forceinline__ uint32_t payload_id(const float4 &v) { return __float_as_uint(v.w); }
__device__ __forceinline__ uint32_t payload_id(const Vec4d &v) { return (uint32_t)__double_as_longlong(v.w); }

// Bead `who` (id, bit 31: the upper z half) arrives in cell `key`: it is counted, and entered in
// the cell's bucket, from which k_move ranks the cell's beads.  A bead that finds its bucket
// full goes into a list of the cell's overflowing beads (its head is valid while its upper word
// is the epoch of this rebuild).
__device__ __forceinline__ void cell_arrive(const KArgs &a, uint32_t key, uint32_t who)
{
    const uint32_t rank = atomicAdd(&a.cnt[key], 1u);
    if (rank < a.bucket_k) {
        a.bucket[(size_t)key * a.bucket_k + rank] = who;
        return;
    }
    const uint32_t node = atomicAdd(&a.over->count, 1u);
    const unsigned long long epoch = (unsigned long long)a.over->epoch + 1ull;
    const unsigned long long prev = atomicExch(&a.over_head[key], epoch << 32 | node);
    a.over_node[node] = make_uint2(who, (prev >> 32) == epoch ? (uint32_t)prev : 0xffffffffu);
}

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr uint32_t SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;
// Up to this many chunks one kernel does the whole prefix sum, each block adding up the counts
// before its own (at most 128 KB, read from L2); above it a first kernel makes the chunks' sums.
// The two launches take about 6 us whatever the size, the one 3 to 4 us up to here.
constexpr uint32_t SCAN_ONE_PASS = 16;

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    uint32_t r = 0;
    if (warp == 0) {
        r = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (lane == 0) sh[0] = r;
    }
    __syncthreads();
    r = sh[0];
    __syncthreads();
    return r;
}

// Chunk `chunk` of the exclusive prefix of cnt[0, n) into start, given what comes before it.
__device__ __forceinline__ void scan_chunk(const uint32_t *__restrict__ cnt, uint32_t n, uint32_t chunk,
                                           uint32_t off, uint32_t *__restrict__ start, uint32_t *sh)
{
    const uint32_t base = chunk * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t tsum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        v[k] = (base + k < n) ? cnt[base + k] : 0u;
        tsum += v[k];
    }
    // Block-wide exclusive scan of the thread totals.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t inc = tsum;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) sh[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
        uint32_t wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        sh[lane] = wi - w;  // exclusive warp offsets
    }
    __syncthreads();
    uint32_t run = off + sh[warp] + (inc - tsum);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        if (base + k < n) start[base + k] = run;
        run += v[k];
    }
}

// What one block of the rebuild does besides: the force pass that produced the counts has
// finished, so every world's t advances (tick) and the next one takes its bricks from a fresh
// queue, room for its lists, and a new epoch of overflow lists.
__device__ __forceinline__ void rebuild_begin(const KArgs &a, int tick)
{
    if (threadIdx.x == 0) {
        *a.brick_next = 0u;
        if (a.list_cursor) a.list_cursor[0] = a.list_cursor[1] = 0ull;
        a.worlds[0].crowded = a.over->count;
        a.over->count = 0u;
        a.over->epoch += 1u;
    }
    if (tick)
        for (uint32_t w = threadIdx.x; w < a.n_worlds; w += blockDim.x) a.worlds[w].t += 1;
}

// Chunk blockIdx.x of the cells' prefix sum, whole (ONE_PASS) or after the chunks' sums.
template <bool ONE_PASS> __device__ __forceinline__ void scan_cells(const KArgs &a, int tick)
{
    __shared__ uint32_t sh[32];
    uint32_t off = 0;
    if (ONE_PASS) {
        if (blockIdx.x == 0) rebuild_begin(a, tick);
        const uint4 *c = (const uint4 *)a.cnt;
        const uint32_t before = blockIdx.x * (SCAN_CHUNK / 4);
#pragma unroll 8
        for (uint32_t k = threadIdx.x; k < before; k += SCAN_THREADS) {
            const uint4 v = c[k];
            off += v.x + v.y + v.z + v.w;
        }
    } else {
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += SCAN_THREADS) off += a.blocksums[b];
    }
    off = block_sum(off, sh);
    scan_chunk(a.cnt, a.n_cells, blockIdx.x, off, a.start, sh);
}

}  // namespace
}  // namespace pdpd
