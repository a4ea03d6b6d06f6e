// Device-side helpers shared by the kernel translation units.
#pragma once

#include <algorithm>
#include <cstdint>

#include "pdpd_internal.h"

namespace pdpd {

// 32-byte aligned FP64 payload element (x, y, z, w).
struct __align__(32) Vec4d {
    double x, y, z, w;
};
struct __align__(16) Vec2d {
    double x, y;
};

// The step kernels are launched so that a kernel's blocks may come up while the one before it
// drains (programmatic dependent launch): each waits for that one to have finished, with its
// writes, before it touches anything.  A step of a small box is three to five kernels of a few
// microseconds, and the gaps between them were a good part of it (9^3 water, 40 steps with the
// read-back: 1.01 -> 0.77 ms).  The short kernels also let the next one's blocks come up at
// once; the force kernels do not, as those blocks would take room on the SMs for nothing
// meanwhile (32^3 polymer box, 100 steps: 3.72 ms without any of this, 3.85 with, 3.54 so).
__device__ __forceinline__ void step_kernel_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void step_kernel_begin()
{
    step_kernel_wait();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_step_kernel(void (*k)(P...), uint32_t grid, uint32_t block, uint32_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, P(args)...);  // (an error is also seen by the caller's cudaGetLastError)
}

// Opt a kernel in to all the dynamic shared memory that a block may have on the current device
// (beside `fixed` bytes of static memory).  The limit belongs to the kernel, for every engine of the
// process: set to the need of one batch, it would refuse the launches of another engine whose batch
// needs more.  What a launch takes (and its occupancy) follows from the bytes it names, not from
// the limit.
inline cudaError_t allow_dynamic_smem(const void *k, size_t fixed = 0)
{
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fixed);
    return e;
}

// Dynamic shared memory with which no more than an even share of `blocks` blocks fits an SM (0 where
// `resident`, those that fit without it, are no more).  The blocks of a force kernel come up while
// the cell-list kernel drains: without it they crowd on the SMs that are free first, and a block
// takes as long as its SM's pipes are shared.  Steps, us, crowded and spread: FP32 bricks, 22^3 of
// density 3 27.4 and 22.7, 24^3 28.5 and 23.8, 25^3 31.8 and 25.0, 16^3 of density 8 37.7 and 29.6;
// variant 6, 22^3 29.9 and 24.3; a thread per bead, 22^3 66.5 and 50.7, 14^3 of density 10 285 and 198;
// the FP64 list kernel, 25^3 87.3 and 81.0.
inline uint32_t spread_smem(uint32_t blocks, int resident, int sm_count, size_t fixed = 0)
{
    int dev = 0, most = 0, opt_in = 0;
    const uint32_t share = (blocks + (uint32_t)sm_count - 1) / (uint32_t)sm_count;
    if (share == 0 || share >= (uint32_t)resident || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&opt_in, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    const int want = most / (int)(share + 1) + 1;  // (one block more would not fit)
    return (uint32_t)std::max(0, std::min(want, opt_in) - (int)fixed);
}

// riscv_mix64_m2 (reference include/dpd/core/hash.hpp:20-30), full 64-bit form.
__device__ __forceinline__ uint64_t mix64_m2(uint64_t x)
{
    const uint64_t C = 0xd392d2a7ull;
    x = x ^ (x >> 32);
    x = x * C;
    x = x ^ (x >> 32);
    x = x * C;
    x = x ^ (x >> 32);
    return x;
}

// get_t_hash (hash.hpp:61-65).
__device__ __forceinline__ uint64_t t_hash(uint32_t t, uint64_t seed)
{
    return mix64_m2(seed + mix64_m2((uint64_t)t));
}

// hash_rng_sym (hash.hpp:81-88): the low 32 bits of mix64_m2((min | max << 32) ^ t_hash),
// evaluated with 32-bit integer operations.  With x = hi:lo and a 32-bit constant C,
// x ^= x >> 32 only changes lo (lo ^= hi), and x *= C gives lo' = lo*C and
// hi' = hi*C + umulhi(lo, C) (mod 2^32).  The final x ^= x >> 32 leaves lo ^ hi in the
// low word, which is all the caller keeps.
__device__ __forceinline__ uint32_t hash_rng_sym(uint32_t th_lo, uint32_t th_hi, uint32_t a,
                                                 uint32_t b)
{
    const uint32_t C = 0xd392d2a7u;
    uint32_t lo = min(a, b) ^ th_lo;
    uint32_t hi = max(a, b) ^ th_hi;
    lo ^= hi;
    uint32_t lo2 = lo * C;
    uint32_t hi2 = hi * C + __umulhi(lo, C);
    lo2 ^= hi2;
    uint32_t lo3 = lo2 * C;
    uint32_t hi3 = hi2 * C + __umulhi(lo2, C);
    return lo3 ^ hi3;
}

// dpd_maths_core::default_hash (dpd_maths_core.hpp:55-79): u = (float)(int32)h * 2^-32,
// uniform on [-0.5, 0.5).
__device__ __forceinline__ float hash_u(uint32_t th_lo, uint32_t th_hi, uint32_t a, uint32_t b)
{
    uint32_t h = hash_rng_sym(th_lo, th_hi, a, b);
    return __int2float_rn((int)h) * 2.3283064365386962890625e-10f;
}

// MIN_DISTANCE_CUTOFF_SQR (dpd_state.hpp:138-139): 1e-9f squared in single precision.
__device__ __forceinline__ float min_dist_sqr_f()
{
    return 0.000000001f * 0.000000001f;
}

__device__ __forceinline__ int wrap_index(int i, int L)
{
    if (i >= L) i -= L;
    if (i < 0) i += L;
    if ((unsigned)i < (unsigned)L) return i;
    i %= L;  // more than one box away
    return i < 0 ? i + L : i;
}

__device__ __forceinline__ void decode_cell(uint32_t local, const int32_t L[3], int &cx, int &cy,
                                            int &cz)
{
    uint32_t yz = (uint32_t)L[1] * (uint32_t)L[2];
    cx = (int)(local / yz);
    uint32_t r = local - (uint32_t)cx * yz;
    cy = (int)(r / (uint32_t)L[2]);
    cz = (int)(r - (uint32_t)cy * (uint32_t)L[2]);
}

}  // namespace pdpd
