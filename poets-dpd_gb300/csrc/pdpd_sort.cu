// Cell-list rebuild: a counting sort of the advanced beads by their new cell.
//
// The step kernels have already counted each bead into its new cell and entered it in the
// cell's bucket (cell_arrive, pdpd_cells.cuh).  Here:
//   1. an exclusive prefix sum of the counts -> start[]: one kernel for up to 32K cells, two
//      above; the launch also holds the bond forces of the next force pass (FP32, and FP64 without
//      pair lists; they need only the advanced positions, so their blocks run beside the few of
//      the prefix sum);
//   2. k_move: each bead ranks itself by (z half, bead id) among its cell's bucket and moves
//      its payload to start[cell] + that rank; the counts are cleared for the next step
//      (after a bin, k_rank and k_gather).
// Small boxes without bond blocks do both in one kernel (k_rebuild_small).
// The result is canonical: cells in index order, beads inside a cell in ascending bead id,
// whatever order the atomics ran in.  That is the order in which the reference's cell lists
// hold beads (naive_dpd_engine_half_step.hpp:276-293), so the FP64 force kernel adds pair
// forces in the reference's order and the engine is deterministic run to run.  The FP32
// engine orders the beads whose cell offset z is >= 0.5 after the lower-half beads of their
// cell, each half in id order, and zlo[cell] counts the lower half, so the half-shell walk can
// skip the far half of an end cell.
// (A first version placed the beads by arrival rank and re-ranked them in a second kernel: five
// launches per step with the bond kernel in front of the force pass.  32^3 polymer box, per
// step: 17 us of sort and 12 us of bonds.)
#include <algorithm>

#include "pdpd_cells.cuh"

namespace pdpd {

uint32_t scan_blocks(uint32_t n_cells)
{
    return (n_cells + SCAN_CHUNK - 1) / SCAN_CHUNK;
}

bool scan_one_pass(uint32_t n_cells)
{
    return scan_blocks(n_cells) <= SCAN_ONE_PASS;
}

// The chunks' sums of cnt[0, n).
__device__ __forceinline__ void reduce_chunk(const uint32_t *__restrict__ cnt, uint32_t n, uint32_t *blocksums)
{
    __shared__ uint32_t sh[32];
    const uint32_t base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (base + k < n) s += cnt[base + k];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) blocksums[blockIdx.x] = s;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_cells_reduce(KArgs a, int tick)
{
    step_kernel_begin();
    if (blockIdx.x == 0) rebuild_begin(a, tick);
    reduce_chunk(a.cnt, a.n_cells, a.blocksums);
}

void launch_cells_reduce(const KArgs &a, int tick, cudaStream_t s)
{
    launch_step_kernel(k_cells_reduce, scan_blocks(a.n_cells), SCAN_THREADS, 0, s, a, tick);
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t *__restrict__ cnt, uint32_t n,
                                                               uint32_t *blocksums)
{
    reduce_chunk(cnt, n, blocksums);
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_final(uint32_t *__restrict__ cnt, uint32_t n,
                                                              const uint32_t *__restrict__ blocksums,
                                                              uint32_t *__restrict__ start)
{
    __shared__ uint32_t sh[32];
    // Offset of this chunk: sum of the preceding chunks' totals.
    uint32_t off = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += blockDim.x) off += blocksums[b];
    off = block_sum(off, sh);
    scan_chunk(cnt, n, blockIdx.x, off, start, sh);
    const uint32_t base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (base + k < n) cnt[base + k] = 0u;
}

// The bead hash carried in the w component of a position payload.
__device__ __forceinline__ uint32_t payload_hash(const float4 &p)
{
    return __float_as_uint(p.w);
}
__device__ __forceinline__ uint32_t payload_hash(const Vec4d &p)
{
    return (uint32_t)__double_as_longlong(p.w);
}

// FP64 positions as FP32 offsets inside their cell (x - floor(x) is exact in FP64, the cell
// being floor(x)), for the force kernel's distance prefilter; the hash rides along.
__device__ __forceinline__ float4 offset_shadow(const Vec4d &p)
{
    return make_float4((float)(p.x - floor(p.x)), (float)(p.y - floor(p.y)), (float)(p.z - floor(p.z)),
                       __uint_as_float(payload_hash(p)));
}

__device__ __forceinline__ uint32_t z_half(const float4 &p) { return p.z >= 0.5f ? 0x80000000u : 0u; }
__device__ __forceinline__ uint32_t z_half(const Vec4d &) { return 0u; }
__device__ __forceinline__ void put_shadow(const KArgs &, uint32_t, const float4 &) {}
__device__ __forceinline__ void put_shadow(const KArgs &a, uint32_t dst, const Vec4d &p) { a.posf[dst] = offset_shadow(p); }

// The place in the new order of bead `me` (id, bit 31: the upper z half) of cell `key`.
__device__ __forceinline__ uint32_t new_place(const KArgs &a, uint32_t key, uint32_t me, const uint32_t *start, uint32_t epoch)
{
    const uint32_t b = start[key], n = start[key + 1] - b;
    const uint32_t m = min(n, a.bucket_k);
    const uint4 *bucket = (const uint4 *)(a.bucket + (size_t)key * a.bucket_k);
    uint32_t rank = 0, lo = 0;
    for (uint32_t k = 0; k < m; k += 4) {
        const uint4 q = bucket[k / 4];
        const uint32_t o[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const bool in = k + u < m;
            rank += in && o[u] < me ? 1u : 0u;
            lo += in && !(o[u] >> 31) ? 1u : 0u;
        }
    }
    if (n > m) {  // the cell's overflowing beads
        const unsigned long long head = a.over_head[key];
        uint32_t node = (uint32_t)(head >> 32) == epoch ? (uint32_t)head : 0xffffffffu;
        while (node != 0xffffffffu) {
            const uint2 o = a.over_node[node];
            rank += o.x < me ? 1u : 0u;
            lo += o.x >> 31 ? 0u : 1u;
            node = o.y;
        }
    }
    if (a.zlo && rank == 0) a.zlo[key] = (uint16_t)min(lo, 0xffffu);
    return b + rank;
}

// Bead s of the old order, its cell, position and velocity given, into its place in the new one.
template <class P>
__device__ __forceinline__ void move_bead(const KArgs &a, uint32_t s, uint32_t key, const P &p, const P &v,
                                          const uint32_t *start, uint32_t epoch, int with_force)
{
    const uint32_t id = payload_id(v);
    const uint32_t dst = new_place(a, key, id | z_half(p), start, epoch);
    ((P *)a.posA)[dst] = p;
    ((P *)a.velA)[dst] = v;
    if (with_force) ((P *)a.frc)[dst] = ((const P *)a.frcB)[s];
    a.ids[dst] = id;
    a.cellg[dst] = key;
    if (!(payload_hash(p) & (1u << 27))) a.slot_of_id[id] = dst;
    put_shadow(a, dst, p);
}

// Bound by memory: reads 8 (cell) + 32 (payload) bytes per bead in the old order, the cell's
// bucket and start, and writes 40 in the new order, which is nearly the old one (a bead moves
// little in a step), so both sides are nearly contiguous.  slot_of_id is kept for polymer beads
// only (monomer bit of the hash clear): the bond forces look partners up through it; the
// codec walks slots and reads ids instead.
template <class P>
__global__ void __launch_bounds__(256) k_move(KArgs a)
{
    step_kernel_begin();
    const uint32_t s = blockIdx.x * 256 + threadIdx.x;
    if (s < a.n_cells) a.cnt[s] = 0u;
    if (s >= a.n_beads) return;
    move_bead(a, s, a.key[s], ((const P *)a.posB)[s], ((const P *)a.velB)[s], a.start, a.over->epoch, 0);
}

// The same after a bin, whose beads are in id order and so far from their places: first each
// bead's slot (ids), then each slot gathers its bead.  Scattered reads cost less than scattered
// writes of the payload (64^3 box in random order: 56 us in k_move, 43 in these two).
template <class P>
__global__ void __launch_bounds__(256) k_rank(KArgs a)
{
    step_kernel_begin();
    const uint32_t s = blockIdx.x * 256 + threadIdx.x;
    if (s < a.n_cells) a.cnt[s] = 0u;
    if (s >= a.n_beads) return;
    const uint32_t half = a.zlo ? z_half(((const P *)a.posB)[s]) : 0u;
    const uint32_t dst = new_place(a, a.key[s], s | half, a.start, a.over->epoch);
    a.ids[dst] = s;
    if (!(a.hash[s] & (1u << 27))) a.slot_of_id[s] = dst;
}

template <class P>
__global__ void __launch_bounds__(256) k_gather(KArgs a)
{
    step_kernel_begin();
    const uint32_t dst = blockIdx.x * 256 + threadIdx.x;
    if (dst >= a.n_beads) return;
    const uint32_t s = a.ids[dst];
    const P p = ((const P *)a.posB)[s];
    ((P *)a.posA)[dst] = p;
    ((P *)a.velA)[dst] = ((const P *)a.velB)[s];
    ((P *)a.frc)[dst] = ((const P *)a.frcB)[s];
    a.cellg[dst] = a.key[s];
    put_shadow(a, dst, p);
}

// The whole rebuild of a small box without bond blocks, by one cluster: every block makes the
// prefix sum for itself, in shared memory, while its first beads' state is on the way; the counts
// are cleared once all blocks have read them.  Bound by the latency of its two rounds of loads.
// The line: cells a block takes in one turn of the prefix sum, and beads it takes in one turn
// (FP64) or three.  Step of water boxes, us, two kernels and one: FP32 4^3 14.1 and 12.8, 9^3
// 15.3 and 14.0, 12^3 (5,184 beads) 16.1 and 15.1, 16^3 (12,288) 17.6 and 16.8; FP64 4^3 29.1
// and 27.4, 8^3 31.8 and 30.4, 10^3 (3,000) 32.9 and 31.1, 12^3 35.3 and 35.1, 14^3 (8,232) 37.7
// and 38.2, 16^3 42.4 and 43.0.
constexpr int SMALL_BLOCKS = 8, SMALL_THREADS = 512;
constexpr uint32_t SMALL_CELLS = SMALL_THREADS * SCAN_ITEMS, SMALL_BEADS = SMALL_BLOCKS * SMALL_THREADS;
template <class P>
__global__ void __cluster_dims__(SMALL_BLOCKS) __launch_bounds__(SMALL_THREADS) k_rebuild_small(KArgs a, int tick, int with_force)
{
    __shared__ uint32_t start[SMALL_CELLS + 1], sh[32];
    step_kernel_begin();
    const uint32_t first = blockIdx.x * SMALL_THREADS + threadIdx.x;
    const uint32_t epoch = a.over->epoch + 1u;
    uint32_t key = 0;
    P p{}, v{};
    if (first < a.n_beads) {
        key = a.key[first];
        p = ((const P *)a.posB)[first];
        v = ((const P *)a.velB)[first];
    }
    scan_chunk(a.cnt, a.n_cells, 0, 0, start, sh);
    if (threadIdx.x == 0) start[a.n_cells] = a.n_beads;
    // every block has read the counts and the epoch
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (uint32_t c = first; c < a.n_cells; c += SMALL_BLOCKS * SMALL_THREADS) {
        a.cnt[c] = 0u;
        a.start[c] = start[c];
    }
    if (blockIdx.x == 0) rebuild_begin(a, tick);
    for (uint32_t s = first; s < a.n_beads;) {
        move_bead(a, s, key, p, v, start, epoch, with_force);
        s += SMALL_BLOCKS * SMALL_THREADS;
        if (s < a.n_beads) {
            key = a.key[s];
            p = ((const P *)a.posB)[s];
            v = ((const P *)a.velB)[s];
        }
    }
}

void launch_scan(uint32_t *cnt, uint32_t n, uint32_t *blocksums, uint32_t *start, cudaStream_t s)
{
    if (n == 0) return;
    const uint32_t nb = scan_blocks(n);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, s>>>(cnt, n, blocksums);
    k_scan_final<<<nb, SCAN_THREADS, 0, s>>>(cnt, n, blocksums, start);
}

int launch_sort(const KArgs &a, int fp64, int tick, int with_force, int bonds, cudaStream_t s)
{
    int n = 0;
    // (the bond blocks look their partners up in the old order: not beside the move)
    const bool bond_blocks = bonds && (fp64 ? !a.list && a.n_bonds + a.n_angles > 0 : a.n_bonded > 0);
    if (a.n_beads > 0 && a.n_beads <= SMALL_BEADS * (fp64 ? 1 : 3) && a.n_cells <= SMALL_CELLS && !bond_blocks) {
        if (fp64) launch_step_kernel(k_rebuild_small<Vec4d>, SMALL_BLOCKS, SMALL_THREADS, 0, s, a, tick, with_force);
        else launch_step_kernel(k_rebuild_small<float4>, SMALL_BLOCKS, SMALL_THREADS, 0, s, a, tick, with_force);
        return 1;
    }
    if (!scan_one_pass(a.n_cells)) {
        launch_cells_reduce(a, tick, s);
        n++;
    }
    n += fp64 ? launch_cells64(a, tick, bonds, s) : launch_cells32(a, tick, bonds, s);
    if (a.n_beads == 0) return n;
    const uint32_t g = (std::max(a.n_beads, a.n_cells) + 255) / 256;
    if (with_force) {
        launch_step_kernel(fp64 ? k_rank<Vec4d> : k_rank<float4>, g, 256, 0, s, a);
        launch_step_kernel(fp64 ? k_gather<Vec4d> : k_gather<float4>, (a.n_beads + 255) / 256, 256, 0, s, a);
        return n + 2;
    }
    launch_step_kernel(fp64 ? k_move<Vec4d> : k_move<float4>, g, 256, 0, s, a);
    return n + 1;
}

__global__ void k_rng_eval(size_t n, const uint32_t *__restrict__ t, const uint64_t *__restrict__ seed,
                           const uint32_t *__restrict__ a, const uint32_t *__restrict__ b,
                           uint32_t *__restrict__ h_out, float *__restrict__ u_out)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t th = t_hash(t[i], seed[i]);
    uint32_t lo = (uint32_t)th, hi = (uint32_t)(th >> 32);
    h_out[i] = hash_rng_sym(lo, hi, a[i], b[i]);
    u_out[i] = hash_u(lo, hi, a[i], b[i]);
}

int launch_rng_eval(size_t n, const uint32_t *t, const uint64_t *seed, const uint32_t *a,
                    const uint32_t *b, uint32_t *h_out, float *u_out, cudaStream_t s)
{
    if (n == 0) return 0;
    k_rng_eval<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, t, seed, a, b, h_out, u_out);
    return 1;
}

size_t payload_bytes(int fp64)
{
    return fp64 ? sizeof(Vec4d) : sizeof(float4);
}

}  // namespace pdpd
