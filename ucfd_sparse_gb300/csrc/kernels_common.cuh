// kernels_common.cuh -- helpers shared by the kernel headers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk_copy.cuh"
#include "kargs.h"

#ifndef UCFD_KNS
#error "UCFD_KNS (kernel namespace) must be defined by the including translation unit"
#endif

#ifndef UCFD_KEXACT
#define UCFD_KEXACT 0
#endif

namespace UCFD_KNS {

constexpr int kBlock = 256;

// Block LU-SGS storage of the two builds.  The exact build keeps the
// reference's arithmetic: off-diagonal blocks J as given, each face's
// product multiplied by fv = face_area * rcp_vol, LU pivots divided by.
// The fast build (FP32 sweeps and the FP64 fused multiply-add mode) folds fv
// into the stored sweep blocks (J fv, formed once per Prepare in FP64) and
// stores reciprocal pivots in the LU diagonal, so a sweep does no division
// and no per-face scaling, and reads no face areas; its block products go
// straight into the right-hand side (one fused multiply-add per entry).
constexpr bool kFold = !UCFD_KEXACT;

__host__ __device__ inline unsigned grid_for(long long n, int block = kBlock) {
    long long g = (n + block - 1) / block;
    return (unsigned)(g > 0 ? g : 1);
}

// Threads per block of a launch with n independent threads (one cell or
// block row each) of type T, at most cap (a tuned launch; 0: none).  A SM
// sub-partition issues one FP64 warp instruction per 64 clocks (2 lanes per
// clock and SM), so the time of a small level is the warps of the busiest
// sub-partition times their instructions: with 256 threads per block a level
// of 1000 cells ran on 4 of the 152 SMs, two warps to a sub-partition.  One
// warp per block while every warp can have a sub-partition to itself; two
// warps per block up to four warps per sub-partition, where whole blocks of
// 256 would leave SMs with one block more than others.  Measured against
// blocks of 256: array LU-SGS step of 32^3 cells (two colours of 16384) 250 ->
// 198 us, natural-order step of 41x36x33 cells (108 levels of at most 1100)
// 6.44 -> 4.04 ms, both FP64.
// FP32 levels that fill the SMs take 128 threads (loop of 128^3 cells 8.99 ms
// with 256, 8.75 with 128, 8.77 with 64); the Krylov kernels ask for 256.
template <typename T>
__host__ inline int spread_block(long long n, int cap) {
    constexpr long long kParts = 4 * 152;  // SM sub-partitions
    const int most = cap > 0 ? cap : (sizeof(T) == 8 ? 64 : 128);
    const long long warps = (n + 31) / 32;
    const int want = warps <= kParts ? 32 : warps <= 4 * kParts ? 64 : most;
    return want < most ? want : most;
}

// x * y rounded on its own (never fused into a following add), so that
// every kernel forms the same term whatever the compiler contracts; with
// contraction off this is the plain product.
__device__ __forceinline__ float mul_rn(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double mul_rn(double x, double y) { return __dmul_rn(x, y); }

// (float)x and (double)x on the integer pipe where the value is a normal
// number of both types or zero: a conversion instruction occupies a SM
// sub-partition's FP64 pipe for 64 clocks, as long as a multiplication, these
// a dozen.  Rounding is to nearest even, as the instruction's; everything
// else (subnormal, overflowing, infinite, NaN) goes to the instruction.
__device__ __forceinline__ float to_float(double x) {
    const unsigned hi = __double2hiint(x), lo = __double2loint(x), mag = hi & 0x7fffffffu;
    unsigned t = __funnelshift_l(lo, hi, 3) - 0xC0000000u;  // exponent - 896 and 23 bits of the mantissa
    t += ((lo << 3) | (t & 1u)) > 0x80000000u ? 1u : 0u;
    t |= hi & 0x80000000u;
    if (mag - 0x38100000u >= 0x0fe00000u) {
        if ((mag | lo) == 0u) t = hi;
        else return (float)x;
    }
    return __uint_as_float(t);
}
__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ double to_double(float x) {
    const unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
    if (mag - 0x00800000u >= 0x7f000000u && mag != 0u) return (double)x;
    const unsigned e = mag ? (mag >> 3) + 0x38000000u : 0u;
    return __hiloint2double((int)(e | (b & 0x80000000u)), (int)(b << 29));
}
__device__ __forceinline__ double to_double(double x) { return x; }
template <typename T, typename S>
__device__ __forceinline__ T convert_to(S x) {
    if constexpr (sizeof(T) == 4) return to_float(x);
    else return to_double(x);
}

// Block-wide sum of a double (blockDim.x multiple of 32, <= 1024); result
// valid in thread 0.
__device__ inline double block_sum(double v) {
    __shared__ double warp_part[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) warp_part[wid] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    v = (threadIdx.x < nw) ? warp_part[threadIdx.x] : 0.0;
    if (wid == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

}  // namespace UCFD_KNS
