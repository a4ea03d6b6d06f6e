// Staging of a brick of cells with its halo and the neighbour walk over it, shared by the FP32
// full-shell force kernels (pdpd_fp32_brick.cuh) and the FP64 list kernel (pdpd_fp64_pairs.cuh).
#pragma once

#include "pdpd_device.cuh"

namespace pdpd {
namespace {

constexpr int SEG_MIN = 9, SEG_MAX = 40;  // walk segments kept per thread: one for each row, or more in dense boxes
constexpr float WALK_R2 = 1.0001f;
constexpr uint32_t SEG_BEADS = 20;      // candidates of one walk segment
constexpr uint32_t SEG_BASE = 0xfffu;   // low 12 bits of a segment: its first pair
constexpr uint32_t FULL_MAX_STAGED = 2 * SEG_BASE;

// A halo coordinate (byte k of the code) as a float: the byte becomes the low mantissa bits of
// 2^23 + v, and the difference of two of these is exact.
template <int K> __device__ __forceinline__ float code_axis(uint32_t code)
{
    return __uint_as_float(__byte_perm(code, 0x4B000000u, 0x7440 + K));
}

// Lower bound of the distance from offset o to the neighbour slab in direction d.
__device__ __forceinline__ float slab_gap(float o, int d)
{
    return d == 0 ? 0.0f : (d < 0 ? o : 1.0f - o);
}

// Two FP32 values per 64-bit register, one instruction for both (sm_100 packed FP32: each half
// rounded as the scalar operation).
__device__ __forceinline__ uint64_t f32x2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The same for all lanes of a warp at t = t0 + lane: the lanes compare the row starts with t0,
// and each lane moves on from the row that this gives.
__device__ __forceinline__ int home_row_near(const uint32_t *rows, int nr, uint32_t t0, uint32_t t)
{
    const int lane = threadIdx.x & 31;
    int r = -1;
    for (int q = 0; q < nr; q += 32)
        r += __popc(__ballot_sync(0xffffffffu, q + lane < nr && rows[q + lane] <= t0));
    while (r + 1 < nr && rows[r + 1] <= t) r++;
    return r;
}

// The in-range bits of the nv <= SEG_BEADS candidates from staged index p (even), the first in
// bit 31: two candidates per packed FP32 instruction, the sign of r^2 - WALK_R2 shifted into
// the mask, four candidates a turn (those past nv are masked out).
__device__ __forceinline__ uint32_t walk_mask(const ulonglong2 *sxy, const uint64_t *szf, uint32_t p,
                                              uint32_t nv, uint64_t nx, uint64_t ny, uint64_t nz, uint64_t m_r2)
{
    const ulonglong2 *xy = sxy + (p >> 1);
    const uint64_t *zf = szf + (p >> 1);
    uint32_t m = 0, done = 0;
#pragma unroll 1
    do {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const ulonglong2 a = xy[q];
            const uint64_t dx = add_f32x2(a.x, nx), dy = add_f32x2(a.y, ny), dz = add_f32x2(zf[q], nz);
            const uint64_t r = fma_f32x2(dz, dz, fma_f32x2(dy, dy, fma_f32x2(dx, dx, m_r2)));
            m = __funnelshift_l((uint32_t)r, m, 1);
            m = __funnelshift_l((uint32_t)(r >> 32), m, 1);
        }
        xy += 2;
        zf += 2;
        done += 4;
    } while (done < nv);
    return (m << (32 - done)) & (uint32_t)((int)0x80000000 >> (int)(nv - 1));
}

// The neighbour walk of one staged home bead at staged index si, offset (ox, oy, oz), halo cell
// `code`: its candidates as segments, 20 candidates' in-range bits (bit 31 the first) over the
// index of their first staged pair, each with at least one bit.
//
// The 9 neighbour rows (dx, dy) in order; a row's 3 cells (dz = -1, 0, +1) are one contiguous
// range of staged beads, a whole end cell left out where its nearest face is >= 1 away.  The
// force kernels are bound by instruction issue, so the walk spends as few instructions per
// candidate as it can: it tests two candidates per packed instruction, on z in brick
// coordinates (no choice of the direction per candidate), and keeps the results as bits instead
// of list entries: 13 instructions for two candidates, where a loop that tested each exactly
// and stored list entries took about 36.  The test is conservative (brick coordinates below 36
// are rounded to 2^-19, so r^2 of a pair in range is off by < 1.2e-5); the exact one follows
// where the candidates are evaluated.  A candidate of a left-out cell and the filler of an odd
// row fail the test.  A lane whose row lies out of reach walks it all the same: the warp takes
// as long as its longest lane.  FP32 force pass of the 128^3 box: 1.14 -> 0.94 ms per step, 186
// -> 140 warp instructions per bead.
//
// segs holds cap segments (cap >= 3) with stride T; flush(n) is called with the n candidates of
// the segments so far when more may not fit, and the walk starts filling them anew.  Returns
// the candidates left in the segments.  PLANES = 3: only the three rows of dx = plane - 1.
//
// TOGETHER: between planes of rows, the lanes of the mask `lanes` (those that walk) flush together
// as soon as one of them has fewer than `spare` segments left: each on its own, in dense
// boxes, they would flush at different rows, one after the other (24^3 boxes, step, us, with nine
// segments each on its own and with brick_segs' number together: density 7 127 and 53, 10 298 and
// 90, 14 571 and 120, 20 1,089 and 277).
template <int T, int PLANES = 1, bool TOGETHER = false, class Flush>
__device__ __forceinline__ int walk_rows(const ulonglong2 *xy, const uint64_t *zf, uint32_t *__restrict__ segs,
                                         int cap, const uint16_t *__restrict__ hstart, int HY, int HZ1,
                                         uint32_t code, uint32_t si, float ox, float oy, float oz, Flush flush,
                                         int plane = 0, uint32_t lanes = 0u, int spare = 3)
{
    const int dlo = PLANES == 3 ? plane - 1 : -1, dhi = PLANES == 3 ? plane - 1 : 1;
    const int hx = (int)(code & 255u), hy = (int)((code >> 8) & 255u), hz = (int)((code >> 16) & 255u);
    const float gzp = 1.0f - oz;
    const float below = WALK_R2 - oz * oz, above = WALK_R2 - gzp * gzp;
    const float zi = -((const float *)zf)[si];
    const uint64_t nz = f32x2(zi, zi), m_r2 = f32x2(-WALK_R2, -WALK_R2);
    const uint16_t *h = hstart + ((hx + dlo) * HY + (hy - 1)) * HZ1 + hz;
    uint32_t *out = segs;
    const uint32_t *const full = segs + (cap - 3) * T;  // room for the first segments of three rows
    int n_cand = 0;
#pragma unroll 1
    for (int ddx = dlo; ddx <= dhi; ddx++) {
        const float gx = slab_gap(ox, ddx), nax = (float)ddx - ox;
        const uint64_t nx = f32x2(nax, nax);
#pragma unroll
        for (int ddy = -1; ddy <= 1; ddy++) {
            const float gy = slab_gap(oy, ddy);
            const float gxy = gx * gx + gy * gy;
            const uint32_t j1 = h[gxy >= above ? 1 : 2];
            uint32_t p = h[gxy >= below ? 0 : -1] & ~1u;
            h += HZ1;
            const float nay = (float)ddy - oy;
            const uint64_t ny = f32x2(nay, nay);
            while (p < j1) {
                uint32_t m = walk_mask(xy, zf, p, min(j1 - p, SEG_BEADS), nx, ny, nz, m_r2);
                if (ddy == 0 && ddx == 0 && si - p < SEG_BEADS) m &= ~(0x80000000u >> (si - p));  // not itself
                if (m) {
                    *out = m | (p >> 1);
                    out += T;
                    n_cand += __popc(m);
                }
                p += SEG_BEADS;
                if (p < j1 && out > full) {
                    flush(n_cand);
                    out = segs;
                    n_cand = 0;
                }
            }
        }
        h += (HY - 3) * HZ1;
        if (ddx < dhi && (TOGETHER ? __any_sync(lanes, out > segs + (cap - spare) * T) : out > full)) {
            flush(n_cand);
            out = segs;
            n_cand = 0;
        }
    }
    return n_cand;
}

// The candidates of walk segments one by one, in order: next() is the staged index of the next
// one.  A segment is read ahead, so that moving on takes no branch (segs has an entry more than
// the walk fills).
template <int T> struct SegReader {
    const uint32_t *segs;
    uint32_t w, ahead;
    __device__ __forceinline__ explicit SegReader(const uint32_t *s) : segs(s), w(0), ahead(s[0]) {}
    __device__ __forceinline__ uint32_t next()
    {
        if (w <= SEG_BASE) {  // no candidate left in the segment
            w = ahead;
            segs += T;
        }
        ahead = segs[0];
        uint32_t b;
        asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(w));
        const uint32_t j = 2 * (w & SEG_BASE) + 31 - b;
        w ^= 1u << b;
        return j;
    }
};

// Halo setup and staging of one brick for the full-shell kernels, block-wide (ends with
// __syncthreads).  Rows (hx, hy) of halo cells, HZ cells each, start at even staged indices (a
// filler far away pads an odd row), so a pair of staged beads never spans two rows:
//   hstart[row * (HZ + 1) + z] = first staged index of halo cell (row, z), the last entry the
//   row's end; hslot[row * HZ + z] = the cell's first slot in the sorted state;
//   home_rows[r] = first home index of home row r, halo_row[r] its halo row; total = staged beads
//   with the fillers.
// If the halo fits (total <= maxb) the beads are staged; else hstart holds nothing of use.  Halo
// coordinates lie in [-1, L] (bricks are cut at the box faces), so each wraps with one
// conditional add or subtract.
//
// pos: the beads' cell offsets by slot; put(j, slot, p, code) keeps what else the
// kernel stages of bead j (code: halo cell hx | hy << 8 | hz << 16, bit 31 for a cell reached
// across the box's faces).
template <int T, class Put>
__device__ __forceinline__ void brick_stage_rows(const KArgs &a, const WorldDev &w, const Brick &br,
                                                 const float4 *__restrict__ pos, uint32_t *home_rows,
                                                 uint16_t *halo_row, uint32_t *staged_total, uint16_t *hstart, uint32_t *hslot,
                                                 uint32_t *rowbase, float *xy, float *zf, uint32_t maxb,
                                                 uint32_t &total, uint32_t &n_home, Put put)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int HX = br.bx + 2, HY = br.by + 2, HZ = br.bz + 2, HZ1 = HZ + 1;
    const int rows = HX * HY;
    const int L0 = w.L[0], L1 = w.L[1], L2 = w.L[2];
    auto row_cell0 = [&](int hx, int hy) {  // global cell (hx, hy, 0) of a halo row
        int gx = br.x0 - 1 + hx, gy = br.y0 - 1 + hy;
        gx += gx < 0 ? L0 : 0;
        gx -= gx >= L0 ? L0 : 0;
        gy += gy < 0 ? L1 : 0;
        gy -= gy >= L1 ? L1 : 0;
        return w.cell_base + ((uint32_t)gx * (uint32_t)L1 + (uint32_t)gy) * (uint32_t)L2;
    };

    // the counts of each row's cells, their prefix in the row, and the row's total: a warp
    // takes as many whole rows as it has lanes for, one lane per cell
    const int group = max(1, 32 / HZ);
    const int sub = lane / HZ, z = lane - sub * HZ;  // (a row of 33 or 34 cells: two turns, below)
    for (int r0 = warp * group; r0 < rows; r0 += (T / 32) * group) {
        const int row = r0 + (HZ > 32 ? 0 : sub);
        const int hx = row / HY, hy = row - hx * HY;
        const bool act = (HZ > 32 || sub < group) && row < rows;
        const uint32_t cell0 = act ? row_cell0(hx, hy) : 0u;
        uint32_t carry = 0, first_home = 0;
        for (int z0 = 0; z0 < HZ; z0 += 32) {
            const int zz = HZ > 32 ? z0 + lane : z;
            const bool on = act && zz < HZ;
            uint32_t n = 0;
            if (on) {
                int gz = br.z0 - 1 + zz;
                gz += gz < 0 ? L2 : 0;
                gz -= gz >= L2 ? L2 : 0;
                const uint32_t s0 = a.start[cell0 + (uint32_t)gz];
                n = a.start[cell0 + (uint32_t)gz + 1] - s0;
                hslot[row * HZ + zz] = s0;
            }
            uint32_t inc = n;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
                if ((HZ > 32 ? lane : z) >= off) inc += y;
            }
            inc += carry;
            if (on) {
                uint16_t *h = hstart + row * HZ1;
                if (zz == 0) h[0] = 0;
                h[zz + 1] = (uint16_t)inc;
                if (zz == HZ - 1) rowbase[row] = inc;
            }
            if (z0 == 0) first_home = __shfl_sync(0xffffffffu, inc, HZ > 32 ? 0 : sub * HZ);
            if (on && zz == br.bz && hx >= 1 && hx <= br.bx && hy >= 1 && hy <= br.by) {
                const int r = (hx - 1) * br.by + (hy - 1);
                home_rows[r] = inc - first_home;
                halo_row[r] = (uint16_t)row;
            }
            carry = HZ > 32 ? __shfl_sync(0xffffffffu, inc, 31) : 0u;
        }
    }
    __syncthreads();
    // warp 0: the rows' staged bases (even) and their total; warp 1: the home rows' prefix
    if (warp < 2) {
        uint32_t *v = warp == 0 ? rowbase : home_rows;
        const int m = warp == 0 ? rows : br.bx * br.by;
        uint32_t carry = 0;
        for (int r0 = 0; r0 < m; r0 += 32) {
            const int r = r0 + lane;
            uint32_t c = r < m ? v[r] : 0u;
            if (warp == 0) c = (c + 1u) & ~1u;
            uint32_t inc = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += y;
            }
            if (r < m) v[r] = carry + inc - c;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) {
            if (warp == 0) *staged_total = carry;
            else home_rows[m] = carry;
        }
    }
    __syncthreads();
    total = *staged_total;
    n_home = home_rows[br.bx * br.by];
    if (total <= maxb) {
        // A row's slots are one run, or at a periodic wrap of z its first or last cell is a run of
        // its own; a bead's halo cell follows from its stored cell.
        const bool wrap_lo = br.z0 == 0, wrap_hi = br.z0 + br.bz == L2;
        int hx = warp / HY, hy = warp - hx * HY;
        for (int row = warp; row < rows; row += T / 32) {
            uint16_t *h = hstart + row * HZ1;
            const uint32_t *hs = hslot + row * HZ;
            const uint32_t base = rowbase[row], len = h[HZ];
            const uint32_t n_lo = wrap_lo ? h[1] : 0u, end_mid = wrap_hi ? h[HZ - 1] : len;
            const uint32_t s_lo = hs[0], s_mid = wrap_lo ? hs[1] - n_lo : s_lo, s_hi = hs[HZ - 1] - end_mid;
            const uint32_t rowcell = (uint32_t)hx | ((uint32_t)hy << 8);
            const bool img = (hx == 0 && br.x0 == 0) || (hx == HX - 1 && br.x0 + br.bx == L0) ||
                             (hy == 0 && br.y0 == 0) || (hy == HY - 1 && br.y0 + br.by == L1);
            const uint32_t row_image = img ? 0x80000000u : 0u;
            const int z_off = 1 - br.z0 - (int)row_cell0(hx, hy);
            for (uint32_t k = lane; k < ((len + 1u) & ~1u); k += 32) {
                const uint32_t j = base + k;
                float4 p = make_float4(1.0e4f, 1.0e4f, 1.0e4f, 0.f);  // the filler
                if (k < len) {
                    const uint32_t slot = k + (k < n_lo ? s_lo : (k < end_mid ? s_mid : s_hi));
                    p = pos[slot];
                    int zz = (int)a.cellg[slot] + z_off;
                    zz = k < n_lo ? 0 : (k < end_mid ? zz : HZ - 1);
                    const uint32_t image = k < n_lo || k >= end_mid ? 0x80000000u : row_image;
                    put(j, slot, p, rowcell | ((uint32_t)zz << 16) | image);
                    p.z += (float)zz;
                }
                float *q = xy + 2 * j - (j & 1u);
                q[0] = p.x;
                q[2] = p.y;
                zf[j] = p.z;
            }
            __syncwarp();
            for (int c = lane; c <= HZ; c += 32) h[c] = (uint16_t)(h[c] + base);
            for (hy += T / 32; hy >= HY; hy -= HY) hx++;
        }
    }
    __syncthreads();
}

}  // namespace
}  // namespace pdpd
