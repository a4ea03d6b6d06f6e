// v2binary snapshot codec on the GPU: the bead records of the BinaryData section of the
// reference's "WorldState v2binary" format (dpd_state_io.hpp:182-247 write_polymer_binary,
// :249-330 read_polymer_binary), encoded straight from the sorted device state.
//
// The section's structure -- per polymer a 16-bit header and optional id deltas -- depends
// only on the topology, so the host writes it once into a device buffer (the layout) with
// the byte offset of every bead's 20-byte record.  A snapshot then fills in the records:
//   position: 3 x uint32, round(x * 65536) (half away from zero), the box side wrapping to 0;
//   v, f: CVec3Half each (cvec3.hpp:132-252): a 5-bit exponent field (e + 15, 0 for the zero
//   vector) and three 9-bit two's-complement mantissas round(c * 2^(8 - e)), low bits first,
//   where e is the largest frexp exponent of the non-zero components (e + 1 if a mantissa
//   rounds to +-256); zero and subnormal components count as zero, e < -14 gives the zero
//   vector, e > 15 or a non-finite component is an error.
// Every step is exact in IEEE double (frexp, ldexp, round), and for the FP32 engine's state in
// single precision, so the bytes equal the reference writer's for the same state.  Records start
// at even offsets (headers are 2 bytes, deltas 4, records 20) and are put together as 16-bit words.
#include <cfloat>

#include "pdpd_device.cuh"

namespace pdpd {

namespace {

// Records of a block of the encoder: small, so that small boxes use many SMs (FP64 box of 2,160
// beads, call: 47.5 us with 512, 34.6 with 64); at 64^3 all of 64 to 512 take the same.
constexpr int V2_TILE = 64;
constexpr uint32_t V2_ERR_VECTOR = 1u;  // non-finite component or magnitude >= 2^15
constexpr uint32_t V2_ERR_BOX = 2u;     // a position outside [0, L)

__device__ __forceinline__ bool cvec3half_encode(const double po[3], uint32_t &word)
{
    double p[3];
    bool any = false;
    int e = -100000;
    for (int i = 0; i < 3; i++) {
        if (!isfinite(po[i])) return false;
        p[i] = fabs(po[i]) < DBL_MIN ? 0.0 : po[i];  // zero and subnormal components
        if (p[i] != 0.0) {
            int ex;
            frexp(p[i], &ex);
            e = max(e, ex);
            any = true;
        }
    }
    if (!any || e < -14) {
        word = 0u;
        return true;
    }
    if (e > 15) return false;
    double fr[3];
    bool over = false;
    for (int i = 0; i < 3; i++) {
        fr[i] = round(ldexp(p[i], 8 - e));
        over |= fabs(fr[i]) == 256.0;
    }
    if (over) {
        e += 1;
        if (e > 15) return false;
        for (int i = 0; i < 3; i++) fr[i] = round(ldexp(p[i], 8 - e));
    }
    word = ((uint32_t)(e + 15) & 0x1Fu) | (((uint32_t)(int)fr[0] & 0x1FFu) << 5) |
           (((uint32_t)(int)fr[1] & 0x1FFu) << 14) | (((uint32_t)(int)fr[2] & 0x1FFu) << 23);
    return true;
}

__device__ __forceinline__ void cvec3half_decode(uint32_t w, double out[3])
{
    const int ex = (int)(w & 0x1Fu);
    for (int i = 0; i < 3; i++) {
        int m = (int)((w >> (5 + 9 * i)) & 0x1FFu);
        if (m >= 256) m -= 512;
        out[i] = ldexp((double)m, ex - 23);
    }
}

// The same for a vector held in single precision: scaling by a power of two and rounding are
// exact there too (a component that underflows rounds to 0 either way; FP32 subnormals are below
// 2^-15, where the vector is zero).
__device__ __forceinline__ bool cvec3half_encode(const float p[3], uint32_t &word)
{
    const float m = fmaxf(fmaxf(fabsf(p[0]), fabsf(p[1])), fabsf(p[2]));
    if (!(isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]))) return false;
    word = 0u;
    if (m < 0x1p-15f) return true;
    int e = (int)(__float_as_uint(m) >> 23) - 126;  // m = f 2^e, f in [0.5, 1)
    if (e > 15) return false;
    float scale = __uint_as_float((uint32_t)(8 - e + 127) << 23);
    float fr[3];
    for (int i = 0; i < 3; i++) fr[i] = roundf(p[i] * scale);
    if (fabsf(fr[0]) == 256.0f || fabsf(fr[1]) == 256.0f || fabsf(fr[2]) == 256.0f) {
        e += 1;
        if (e > 15) return false;
        scale *= 0.5f;
        for (int i = 0; i < 3; i++) fr[i] = roundf(p[i] * scale);
    }
    word = ((uint32_t)(e + 15) & 0x1Fu) | (((uint32_t)(int)fr[0] & 0x1FFu) << 5) |
           (((uint32_t)(int)fr[1] & 0x1FFu) << 14) | (((uint32_t)(int)fr[2] & 0x1FFu) << 23);
    return true;
}

__device__ __forceinline__ void load_words(const uint8_t *src, uint32_t w[5])
{
    const uint16_t *s = reinterpret_cast<const uint16_t *>(src);
    for (int k = 0; k < 5; k++) w[k] = (uint32_t)s[2 * k] | ((uint32_t)s[2 * k + 1] << 16);
}

// The five words of slot s's record; the error bits.
template <int FP64> __device__ __forceinline__ uint32_t encode_record(const KArgs &a, const WorldDev &w, uint32_t s,
                                                                      uint32_t word[5])
{
    uint32_t bad = 0;
    if (FP64) {
        const Vec4d p = ((const Vec4d *)a.posA)[s], vv = ((const Vec4d *)a.velA)[s],
                    ff = ((const Vec4d *)a.frc)[s];
        const double x[3] = {p.x, p.y, p.z}, v[3] = {vv.x, vv.y, vv.z}, f[3] = {ff.x, ff.y, ff.z};
        for (int d = 0; d < 3; d++) {
            const double side = (double)w.L[d] * 65536.0;
            double rr = round(x[d] * 65536.0);
            if (rr == side) rr = 0.0;
            if (!(rr >= 0.0 && rr < side)) {
                bad |= V2_ERR_BOX;
                rr = 0.0;
            }
            word[d] = (uint32_t)rr;
        }
        if (!cvec3half_encode(v, word[3])) bad |= V2_ERR_VECTOR;
        if (!cvec3half_encode(f, word[4])) bad |= V2_ERR_VECTOR;
    } else {
        const float4 p = ((const float4 *)a.posA)[s], vv = ((const float4 *)a.velA)[s],
                     ff = ((const float4 *)a.frc)[s];
        int c[3];
        decode_cell(a.cellg[s] - w.cell_base, w.L, c[0], c[1], c[2]);
        const float o[3] = {p.x, p.y, p.z}, v[3] = {vv.x, vv.y, vv.z}, f[3] = {ff.x, ff.y, ff.z};
        for (int d = 0; d < 3; d++) {
            // x = c + o: round(x 65536) = c 65536 + round(o 65536), both products exact
            uint32_t rr = (uint32_t)c[d] * 65536u;
            if (o[d] >= 0.0f && o[d] < 1.0f) rr += (uint32_t)roundf(o[d] * 65536.0f);
            else bad |= V2_ERR_BOX;
            word[d] = rr == (uint32_t)w.L[d] * 65536u ? 0u : rr;
        }
        if (!cvec3half_encode(v, word[3])) bad |= V2_ERR_VECTOR;
        if (!cvec3half_encode(f, word[4])) bad |= V2_ERR_VECTOR;
    }
    return bad;
}

// The section of V2_TILE records, in record order: each thread gathers its bead (inv: the slot of
// each global bead id), puts its record and the structure bytes before it together in shared
// memory, and the block writes the tile's run of bytes back in 16-byte words (the structure bytes
// unchanged).  One thread per slot, writing its record as ten 16-bit words wherever it lies and
// encoding FP32 values in FP64, took 194 us for the 64^3 box against 25 us.
template <int FP64>
__global__ void __launch_bounds__(V2_TILE) k_v2_encode(KArgs a, uint32_t world, uint32_t n, const uint2 *__restrict__ rec,
                                                       const uint32_t *__restrict__ inv, uint8_t *buf,
                                                       uint32_t *err)
{
    extern __shared__ __align__(16) uint8_t s_run[];
    step_kernel_wait();
    const WorldDev &w = a.worlds[world];
    const uint32_t r0 = blockIdx.x * V2_TILE, r1 = min(n, r0 + V2_TILE), r = r0 + threadIdx.x;
    const uint32_t b0 = r0 ? rec[r0 - 1].y + 20u : 0u, b1 = rec[r1 - 1].y + 20u;
    const uint32_t pad = (uint32_t)((uintptr_t)(buf + b0) & 15u);  // the run's place in its first 16-byte word
    if (r < r1) {
        const uint2 me = rec[r];
        const uint32_t gap = r ? rec[r - 1].y + 20u : 0u;  // the structure bytes [gap, me.y)
        uint32_t word[5];
        const uint32_t bad = encode_record<FP64>(a, w, inv[w.bead_base + me.x], word);
        if (bad) atomicOr(err, bad);
        uint16_t *out = reinterpret_cast<uint16_t *>(s_run + pad + (gap - b0));
        for (uint32_t k = gap; k < me.y; k += 2) *out++ = *reinterpret_cast<const uint16_t *>(buf + k);
        for (int k = 0; k < 5; k++) {
            *out++ = (uint16_t)(word[k] & 0xFFFFu);
            *out++ = (uint16_t)(word[k] >> 16);
        }
    }
    __syncthreads();
    uint8_t *base = buf + b0 - pad;  // 16-byte aligned
    const uint32_t end = pad + (b1 - b0);
    for (uint32_t k = 16 * threadIdx.x; k < end; k += 16 * V2_TILE) {
        if (k >= pad && k + 16 <= end) {
            *reinterpret_cast<uint4 *>(base + k) = *reinterpret_cast<const uint4 *>(s_run + k);
        } else {
            for (uint32_t q = max(k, pad); q < min(k + 16, end); q += 2)
                *reinterpret_cast<uint16_t *>(base + q) = *reinterpret_cast<const uint16_t *>(s_run + q);
        }
    }
}

// Decode one world's records into the id-ordered staging rows (x, v, f per bead).
__global__ void k_v2_decode(KArgs a, uint32_t world, uint32_t n, const uint8_t *__restrict__ buf,
                            const uint32_t *__restrict__ off, double *__restrict__ staging,
                            uint32_t *err)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const WorldDev &w = a.worlds[world];
    uint32_t word[5];
    load_words(buf + off[i], word);
    double *row = staging + 9 * (size_t)(w.bead_base + i);
    for (int d = 0; d < 3; d++) {
        const double x = ldexp((double)word[d], -16);
        if (!(x < (double)w.L[d])) atomicOr(err, V2_ERR_BOX);
        row[d] = x;
    }
    cvec3half_decode(word[3], row + 3);
    cvec3half_decode(word[4], row + 6);
}

}  // namespace

int launch_v2_encode(const KArgs &a, int fp64, uint32_t world, uint32_t n, const uint2 *rec, const uint32_t *inv,
                     uint8_t *buf, uint32_t *err, cudaStream_t s)
{
    if (n == 0) return 0;
    const uint32_t g = (n + V2_TILE - 1) / V2_TILE;
    const uint32_t smem = V2_TILE * 30 + 32;  // a record, its delta and its polymer's header and delta
    if (fp64)
        launch_step_kernel(k_v2_encode<1>, g, V2_TILE, smem, s, a, world, n, rec, inv, buf, err);
    else
        launch_step_kernel(k_v2_encode<0>, g, V2_TILE, smem, s, a, world, n, rec, inv, buf, err);
    return 1;
}

int launch_v2_decode(const KArgs &a, uint32_t world, uint32_t n, const uint8_t *buf,
                     const uint32_t *off, double *staging, uint32_t *err, cudaStream_t s)
{
    if (n == 0) return 0;
    k_v2_decode<<<(n + 255) / 256, 256, 0, s>>>(a, world, n, buf, off, staging, err);
    return 1;
}

}  // namespace pdpd
