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
template <typename T>
__host__ inline int spread_block(long long n, int cap) {
    constexpr long long kParts = 4 * 152;  // SM sub-partitions
    const int most = cap > 0 ? cap : (sizeof(T) == 8 ? 64 : 256);
    const long long warps = (n + 31) / 32;
    const int want = warps <= kParts ? 32 : warps <= 4 * kParts ? 64 : most;
    return want < most ? want : most;
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
