// launchers.cuh -- definitions of the launch.h declarations for the
// namespace UCFD_KNS; included once by each kernel translation unit.
#pragma once

#include "launch.h"
#include "kernels_lusgs.cuh"
#include "kernels_blusgs.cuh"
#include "kernels_krylov.cuh"
#include "kernels_adjoint.cuh"
#include "ucfd_internal.h"

namespace UCFD_KNS {

// ---- adjoint of the colored LU-SGS step --------------------------------------
template <typename T>
void adj_upper(const ::ucfd::AdjArgs &a, int nfv, int ndims, T gamma, T pmin, const T *fnv, const T *vec,
               const T *fspr, const T *upts, const T *diag, const T *dub, const T *dq, const T *gdq, T *qbar, T *wbuf,
               T *dbar, T *gfspr, cudaStream_t s) {
    const int n = a.t1 - a.t0;
    if (n <= 0) return;
    const int block = spread_block<T>(n, 0);
    if (nfv == 5 && ndims == 3)
        return adj_upper_kernel<T, 5, 3><<<grid_for(n, block), block, 0, s>>>(a, gamma, pmin, fnv, vec, fspr, upts, diag,
                                                                              dub, dq, gdq, qbar, wbuf, dbar, gfspr);
    if (nfv == 4 && ndims == 2)
        return adj_upper_kernel<T, 4, 2><<<grid_for(n, block), block, 0, s>>>(a, gamma, pmin, fnv, vec, fspr, upts, diag,
                                                                              dub, dq, gdq, qbar, wbuf, dbar, gfspr);
    ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "adjoint built for nfvars/ndims 5/3 and 4/2 only");
}

template <typename T>
void adj_lower(const ::ucfd::AdjArgs &a, int nfv, int ndims, T gamma, T pmin, T factor, const T *fnv, const T *vec,
               const T *fspr, const T *dt, const T *upts, const T *diag, const T *dub, const T *qbar, T *wbuf,
               const T *dbar, T *grhs, T *gdt, T *gfspr, cudaStream_t s) {
    const int n = a.t1 - a.t0;
    if (n <= 0) return;
    const int block = spread_block<T>(n, 0);
    if (nfv == 5 && ndims == 3)
        return adj_lower_kernel<T, 5, 3><<<grid_for(n, block), block, 0, s>>>(
            a, gamma, pmin, factor, fnv, vec, fspr, dt, upts, diag, dub, qbar, wbuf, dbar, grhs, gdt, gfspr);
    if (nfv == 4 && ndims == 2)
        return adj_lower_kernel<T, 4, 2><<<grid_for(n, block), block, 0, s>>>(
            a, gamma, pmin, factor, fnv, vec, fspr, dt, upts, diag, dub, qbar, wbuf, dbar, grhs, gdt, gfspr);
    ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "adjoint built for nfvars/ndims 5/3 and 4/2 only");
}

// ---- scalar LU-SGS ---------------------------------------------------------
template <typename T>
void face_list_geo(long long E, long long ld, int ndims, const int *q, const T *nrm, const T *fa, const T *rv,
                   T *geo, cudaStream_t s) {
    if (E <= 0) return;
    const long long g = (E + kBlock - 1) / kBlock;
    face_list_geo_kernel<T><<<(unsigned)(g < 65535 * 16 ? g : 65535 * 16), kBlock, 0, s>>>(E, ld, ndims, q, nrm, fa,
                                                                                          rv, geo);
}

void face_fv(long long N, int P, const double *fa, const double *rv, double *fv, cudaStream_t s) {
    const long long n = (long long)P * N;
    if (n <= 0) return;
    const long long g = (n + kBlock - 1) / kBlock;
    face_fv_kernel<<<(unsigned)(g < 65535 * 16 ? g : 65535 * 16), kBlock, 0, s>>>(N, P, fa, rv, fv);
}

void pack_geo4(long long N, int P, int ndims, const float *nrm, const float *fa, const float *rv, void *geo4,
               cudaStream_t s) {
    const long long n = (long long)P * N;
    if (n <= 0) return;
    const long long g = (n + kBlock - 1) / kBlock;
    pack_geo4_kernel<<<(unsigned)(g < 65535 * 16 ? g : 65535 * 16), kBlock, 0, s>>>(N, P, ndims, nrm, fa, rv,
                                                                                   static_cast<float4 *>(geo4));
}

void pack_lam2(long long n, const float *lam, const float *tlam, void *lam2, cudaStream_t s) {
    if (n <= 0) return;
    const long long g = (n + kBlock - 1) / kBlock;
    pack_lam2_kernel<<<(unsigned)(g < 65535 * 16 ? g : 65535 * 16), kBlock, 0, s>>>(n, lam, tlam,
                                                                                   static_cast<float2 *>(lam2));
}

// A sweep kernel of one level; in FP32 a chained level as a programmatic
// dependent of the previous one (in FP64 waiting blocks would crowd onto the
// SMs that run out of work first, see the block sweeps).
template <typename T>
static void sweep_launch(void (*kern)(::ucfd::ScalarSweepArgs<T>), const ::ucfd::ScalarSweepArgs<T> &a, long long n,
                         int block, cudaStream_t s) {
    ::ucfd::ScalarSweepArgs<T> b = a;
    if (sizeof(T) == 8) b.chained = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_for(n, block));
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = b.chained ? 1 : 0;
    UCFD_CUDA(cudaLaunchKernelEx(&cfg, kern, b));
}

template <typename T, int NV, int NFV, int NDIMS, bool RANS>
static void sweep_go(const ::ucfd::ScalarSweepArgs<T> &a, int block, cudaStream_t s) {
    const long long n = a.t1 - a.t0;
    if (n <= 0) return;
    if (a.facelist) {
        constexpr int DNV = RANS ? NV - NFV : NFV;
        ::ucfd::ScalarSweepArgs<T> b = a;
        if (b.cpb <= 0 || b.cpb > block) b.cpb = block / 3 > 0 ? block / 3 : 1;
        const size_t smem = (size_t)b.cpb * (a.nface > 0 ? a.nface : 1) * DNV * sizeof(T);
        if (smem > 48 * 1024) ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "face-list sweep: %zu bytes of shared memory", smem);
        scalar_sweep_faces_kernel<T, NV, NFV, NDIMS, RANS><<<grid_for(n, b.cpb), block, smem, s>>>(b);
        return;
    }
    if (a.pair && a.nface <= 6) {
        if (a.regcap == 4)
            scalar_sweep_pair_kernel<T, NV, NFV, NDIMS, RANS, 4><<<grid_for(2 * n, block), block, 0, s>>>(a);
        else
            scalar_sweep_pair_kernel<T, NV, NFV, NDIMS, RANS, 1><<<grid_for(2 * n, block), block, 0, s>>>(a);
        return;
    }
    if (a.regcap == 4)
        sweep_launch<T>(scalar_sweep_kernel<T, NV, NFV, NDIMS, RANS, 4>, a, n, block, s);
    else if (a.regcap == 3)
        sweep_launch<T>(scalar_sweep_kernel<T, NV, NFV, NDIMS, RANS, 3>, a, n, block, s);
    else
        sweep_launch<T>(scalar_sweep_kernel<T, NV, NFV, NDIMS, RANS, 1>, a, n, block, s);
}

// Both systems in one launch per level (one thread per cell; the register
// caps of the single-system kernels).
template <typename T, int NV, int NFV, int NDIMS>
static void sweep_both_go(const ::ucfd::ScalarSweepArgs<T> &a, int block, cudaStream_t s) {
    const long long n = a.t1 - a.t0;
    if (n <= 0) return;
    if (a.facelist || a.pair)
        ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "both-system sweep: one thread per cell only");
    if (a.regcap == 4)
        sweep_launch<T>(scalar_sweep_both_kernel<T, NV, NFV, NDIMS, 4>, a, n, block, s);
    else if (a.regcap == 3)
        sweep_launch<T>(scalar_sweep_both_kernel<T, NV, NFV, NDIMS, 3>, a, n, block, s);
    else
        sweep_launch<T>(scalar_sweep_both_kernel<T, NV, NFV, NDIMS, 1>, a, n, block, s);
}

// FP64 levels of at most this many cells take scalar_sweep_lanes_kernel: with
// 4 / 8 pairs of lanes per cell.  One warp holds 4 / 2 cells and issues about
// 95 FP64 instructions, against 480 (three active faces) to 900 (six) for a
// warp of 32 cells with one thread per cell, so the lanes cost more pipe time
// per cell and win while the sub-partitions (608) have few warps each.
// Measured: natural-order FP64 step of 41x36x33 cells (108 levels of at most
// 1100 cells, three active faces) 4.04 ms with one thread per cell in
// blocks of 32, 0.91 ms with lanes chained by dependent launches.  A lower +
// upper pair of two colours, lanes / one thread per cell, exact mode:
//   quadrilaterals (4): 4608 cells a colour 26.7 / 45.1 us, 8192 41.0 / 45.1,
//     10368 55.3 / 47.1, 12800 59.5 / 45.2;
//   hexahedra (8): 4000 47.1 / 69.6 us, 6083 67.9 / 71.7, 6912 77.8 / 69.7.
// (FMA mode: 8192 36.9 / 43.0, 10368 49.0 / 44.6; 6083 61.4 / 63.6, 6912 67.6 / 63.5.)
constexpr int kLanesCells4 = 8192, kLanesCells8 = 6144;

template <int NV, int NFV, int NDIMS, int SYS>
static void sweep_lanes_go(const ::ucfd::ScalarSweepArgs<double> &a, int gf, cudaStream_t s) {
    const long long n = a.t1 - a.t0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_for(n * 2 * gf, kLanesThreads), SYS == 2 ? 2 : 1);
    cfg.blockDim = dim3(kLanesThreads);
    cfg.stream = s;
    // the next level's launch may start while this level runs
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.chained ? 1 : 0;
    if (gf == 4) UCFD_CUDA(cudaLaunchKernelEx(&cfg, scalar_sweep_lanes_kernel<NV, NFV, NDIMS, SYS, 4>, a));
    else UCFD_CUDA(cudaLaunchKernelEx(&cfg, scalar_sweep_lanes_kernel<NV, NFV, NDIMS, SYS, 8>, a));
}

// Larger FP64 levels with rows of at most 8 faces: one thread per active face
// of a block's cells, whatever the launch variant's register cap.  Up to
// kPackedMin cells one thread per cell has a sub-partition's FP64 pipe nearly
// to itself, and the lists' barriers cost more than idle lanes (32^3 cells
// in two colours of 16384: 191 us a step against 197).  What the lists gain
// are the idle lanes of uneven cells.  Lower + upper pair of the greedy
// colours of permuted hexahedra, exact mode, with the line at 8192 / 16384 /
// 32768 / no lists: 40^3 cells (colours up to 20105) 223 / 225 / 250 / 250 us,
// 48^3 (34692) 283 / 287 / 303 / 328, 56^3 (55242) 387 / 387 / 399 / 463, 64^3
// (81893) 609 / 608 / 607 / 721.  Where every cell of a level has the same
// faces (a checkerboard) there is nothing to gain and up to 2 % to lose:
// colours of 19652 cells 104 us with lists, 103 without; 108000 395 and 385.
constexpr int kPackedMin = 16384;

template <int NV, int NFV, int NDIMS, int SYS>
static void sweep_packed_go(const ::ucfd::ScalarSweepArgs<double> &a, cudaStream_t s) {
    const unsigned g = grid_for(a.t1 - a.t0, 64);
    if (a.nface <= 6) scalar_sweep_packed_kernel<NV, NFV, NDIMS, SYS, 6><<<g, 64, 0, s>>>(a);
    else scalar_sweep_packed_kernel<NV, NFV, NDIMS, SYS, 8><<<g, 64, 0, s>>>(a);
}

// Pairs of lanes per cell for a level of this kind, 0: another kernel.
static int sweep_lanes(const ::ucfd::ScalarSweepArgs<double> &a) {
    const long long n = a.t1 - a.t0;
    if (a.pair || a.facelist || a.nface > 8 || n <= 0) return 0;
    const int most = a.max_active > 0 ? a.max_active : a.nface;
    if (most <= 4) return n <= kLanesCells4 ? 4 : 0;
    return n <= kLanesCells8 ? 8 : 0;
}
static int sweep_lanes(const ::ucfd::ScalarSweepArgs<float> &) { return 0; }

// rans: 0 mean-flow system, 1 turbulence system, 2 both in one launch.
template <typename T>
void scalar_sweep(const ::ucfd::ScalarSweepArgs<T> &a, int nv, int nfv, int ndims, int rans,
                  int block, cudaStream_t s) {
    if (a.facelist) block = block > 0 ? block : kBlock;
    else block = spread_block<T>(a.pair ? 2ll * (a.t1 - a.t0) : a.t1 - a.t0, block);
    const int gf = sweep_lanes(a);
    const bool packed = sizeof(T) == 8 && gf == 0 && !a.pair && !a.facelist && a.nface <= 8 &&
                        a.t1 - a.t0 > kPackedMin;
#define UCFD_SW(NV, NFV, ND)                                                   \
    if (nv == NV && nfv == NFV && ndims == ND) {                               \
        if constexpr (sizeof(T) == 8) {                                        \
            if (packed && rans == 0) return sweep_packed_go<NV, NFV, ND, 0>(a, s); \
            if constexpr (NV > NFV) {                                          \
                if (packed && rans == 1) return sweep_packed_go<NV, NFV, ND, 1>(a, s); \
                if (packed) return sweep_packed_go<NV, NFV, ND, 2>(a, s);      \
            }                                                                  \
            if (gf > 0 && rans == 0) return sweep_lanes_go<NV, NFV, ND, 0>(a, gf, s); \
            if constexpr (NV > NFV) {                                          \
                if (gf > 0 && rans == 1) return sweep_lanes_go<NV, NFV, ND, 1>(a, gf, s); \
                if (gf > 0) return sweep_lanes_go<NV, NFV, ND, 2>(a, gf, s);   \
            }                                                                  \
        }                                                                      \
        if (rans == 2) {                                                       \
            if constexpr (NV > NFV) return sweep_both_go<T, NV, NFV, ND>(a, block, s); \
        } else if (rans) {                                                     \
            if constexpr (NV > NFV) return sweep_go<T, NV, NFV, ND, true>(a, block, s); \
        } else {                                                               \
            return sweep_go<T, NV, NFV, ND, false>(a, block, s);               \
        }                                                                      \
    }
    UCFD_SW(5, 5, 3)
    UCFD_SW(6, 5, 3)
    UCFD_SW(7, 5, 3)
    UCFD_SW(4, 4, 2)
    UCFD_SW(5, 4, 2)
    UCFD_SW(6, 4, 2)
#undef UCFD_SW
    ::ucfd::fail(UCFD_ERR_UNSUPPORTED,
                 "scalar sweep for nvars=%d nfvars=%d ndims=%d (%s) is not built (supported: "
                 "ndims 3 with nfvars 5, ndims 2 with nfvars 4, up to 2 turbulence variables)",
                 nv, nfv, ndims, rans ? "RANS" : "NS");
}

template <typename T, int NV, int NFV, int NDIMS, bool RANS, int MINB, bool BOTH = false>
static void persistent_minb_go(const ::ucfd::ScalarSweepArgs<T> &a, const int *lev_off, int nlev, unsigned *bar,
                               int *err, long long max_spin, cudaStream_t s) {
    auto kern = scalar_sweep_persistent_kernel<T, NV, NFV, NDIMS, RANS, MINB, BOTH>;
    static int grid = 0;  // per instantiation: blocks that fit co-resident
    if (!grid) {
        int per_sm = 0, dev = 0, sms = 0;
        UCFD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, 0));
        UCFD_CUDA(cudaGetDevice(&dev));
        UCFD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        grid = per_sm * sms;
        if (grid <= 0) ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "persistent sweep kernel does not fit on the device");
    }
    ::ucfd::ScalarSweepArgs<T> aa = a;
    void *args[] = {(void *)&aa, (void *)&lev_off, (void *)&nlev, (void *)&bar, (void *)&err, (void *)&max_spin};
    UCFD_CUDA(cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(kBlock), args, 0, s));
}

template <typename T, int NV, int NFV, int NDIMS, bool RANS, bool BOTH = false>
static void persistent_go(const ::ucfd::ScalarSweepArgs<T> &a, const int *lev_off, int nlev, unsigned *bar,
                          int *err, long long max_spin, cudaStream_t s) {
    if (a.regcap == 4)
        persistent_minb_go<T, NV, NFV, NDIMS, RANS, 4, BOTH>(a, lev_off, nlev, bar, err, max_spin, s);
    else if (a.regcap == 3)
        persistent_minb_go<T, NV, NFV, NDIMS, RANS, 3, BOTH>(a, lev_off, nlev, bar, err, max_spin, s);
    else
        persistent_minb_go<T, NV, NFV, NDIMS, RANS, 2, BOTH>(a, lev_off, nlev, bar, err, max_spin, s);
}

// Whole sweep (all nlev levels) as one cooperative launch with a bounded
// grid barrier between levels; lev_off is a device array.
template <typename T>
void scalar_sweep_persistent(const ::ucfd::ScalarSweepArgs<T> &a, int nv, int nfv, int ndims, int rans,
                             const int *lev_off, int nlev, unsigned *bar, int *err, long long max_spin,
                             cudaStream_t s) {
#define UCFD_PSW(NV, NFV, ND)                                                                              \
    if (nv == NV && nfv == NFV && ndims == ND) {                                                           \
        if (rans == 2) {                                                                                   \
            if constexpr (NV > NFV) return persistent_go<T, NV, NFV, ND, true, true>(a, lev_off, nlev, bar, \
                                                                                      err, max_spin, s);   \
        } else if (rans) {                                                                                 \
            if constexpr (NV > NFV) return persistent_go<T, NV, NFV, ND, true>(a, lev_off, nlev, bar, err, \
                                                                                max_spin, s);              \
        } else {                                                                                           \
            return persistent_go<T, NV, NFV, ND, false>(a, lev_off, nlev, bar, err, max_spin, s);          \
        }                                                                                                  \
    }
    UCFD_PSW(5, 5, 3)
    UCFD_PSW(6, 5, 3)
    UCFD_PSW(7, 5, 3)
    UCFD_PSW(4, 4, 2)
    UCFD_PSW(5, 4, 2)
    UCFD_PSW(6, 4, 2)
#undef UCFD_PSW
    ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "persistent sweep for nvars=%d nfvars=%d ndims=%d is not built", nv, nfv,
                 ndims);
}

template <typename T>
void legacy_pre(int neles, int nface, T factor, const T *fnorm_vol, const T *dt, T *diag,
                const T *fspr, cudaStream_t s) {
    if (neles <= 0) return;
    legacy_pre_kernel<T><<<grid_for(neles), kBlock, 0, s>>>(neles, nface, factor, fnorm_vol, dt, diag, fspr);
}

template <typename T>
void legacy_update(int neles, int k0, int k1, T *upts, const T *rhs, cudaStream_t s) {
    if (neles <= 0 || k1 <= k0) return;
    legacy_update_kernel<T><<<grid_for(neles), kBlock, 0, s>>>(neles, k0, k1, upts, rhs);
}

template <typename T>
void fs_lusgs_pack(int neles, int nvars, int nfvars, long long N, double turb_factor, double a0,
                   const int *cell_ids, const int *iperm, const double *upts, const double *rhs,
                   const double *dt, const double *dsrc, T *u, T *du, T *diag, cudaStream_t s) {
    if (neles <= 0) return;
    fs_lusgs_pack_kernel<T><<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, nfvars, N, turb_factor, a0,
                                                                cell_ids, iperm, upts, rhs, dt, dsrc, u,
                                                                du, diag);
}

// Two-pass Pack (records, then the arrays), nvars 4 .. 7; false: not built for
// this nvars.  rec holds N records of pack_record_words words.
template <typename T>
int pack_record_words(int nvars) { return pack_words<T>(nvars); }

template <typename T>
bool fs_lusgs_pack_records(int neles, int nvars, int nfvars, long long N, double turb_factor, double a0,
                           const int *cell_ids, const int *iperm, const double *upts, const double *rhs,
                           const double *dt, const double *dsrc, int stamp, T *rec, T *u, T *du, T *diag, T *base,
                           T *rhs0, T *ulo, cudaStream_t s) {
#define UCFD_PACK(NV)                                                                                            \
    case NV:                                                                                                     \
        fs_lusgs_pack_records_kernel<T, NV><<<grid_for(neles), kBlock, 0, s>>>(                                  \
            neles, nfvars, turb_factor, a0, cell_ids, iperm, upts, rhs, dt, dsrc, stamp, rec);                   \
        fs_lusgs_unpack_kernel<T, NV><<<grid_for(N, 128), 128, 0, s>>>(N, stamp, rec, u, du, diag, base, rhs0,   \
                                                                      ulo);                                      \
        return true;
    switch (nvars) {
        UCFD_PACK(4)
        UCFD_PACK(5)
        UCFD_PACK(6)
        UCFD_PACK(7)
        default: return false;
    }
#undef UCFD_PACK
}

template <typename T>
void fs_lusgs_update(int neles, int nvars, long long N, const int *cell_ids, const int *iperm,
                     const T *du, double *upts, int assign, cudaStream_t s) {
    if (neles <= 0) return;
    fs_lusgs_update_kernel<T><<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, N, cell_ids, iperm, du, upts, assign);
}

template <typename T>
void fs_lusgs_prepare(long long N, int maxdeg, int nv0, int nv1, T kappa, const int *nei,
                      const T *fa, const T *rv, const T *lam, const T *base, T *diag, cudaStream_t s) {
    if (N <= 0) return;
    fs_lusgs_prepare_kernel<T><<<grid_for(N), kBlock, 0, s>>>(N, maxdeg, nv0, nv1, kappa, nei, fa, rv, lam,
                                                              base, diag);
}

template <typename T>
void fs_lusgs_prepare_both(long long N, int maxdeg, int nfv, int nv, T kappa, const int *nei, const T *fa,
                           const T *rv, const T *lam, const T *tlam, const T *base, T *diag, cudaStream_t s) {
    if (N <= 0) return;
    fs_lusgs_prepare_both_kernel<T><<<grid_for(N), kBlock, 0, s>>>(N, maxdeg, nfv, nv, kappa, nei, fa, rv, lam,
                                                                   tlam, base, diag);
}

template <typename T>
void fs_lusgs_gather_prepare(long long N, int maxdeg, int nv0, int nfv, int nv1, T kappa, const int *slot, const T *fa,
                             const T *rv, const double *lamf, const double *tlamf, T *lam, T *tlam, void *lam2,
                             T *diag, cudaStream_t s) {
    if (N <= 0) return;
    const unsigned g = grid_for(N);
    if (tlamf)
        fs_lusgs_gather_prepare_kernel<T, true><<<g, kBlock, 0, s>>>(N, maxdeg, nv0, nfv, nv1, kappa, slot, fa, rv, lamf,
                                                                     tlamf, lam, tlam, static_cast<float2 *>(lam2),
                                                                     diag);
    else
        fs_lusgs_gather_prepare_kernel<T, false><<<g, kBlock, 0, s>>>(N, maxdeg, nv0, nfv, nv1, kappa, slot, fa, rv,
                                                                      lamf, nullptr, lam, nullptr, nullptr, diag);
}

template <typename Td>
void gather_idx(long long n, const int *idx, const double *src, Td *dst, cudaStream_t s) {
    if (n <= 0) return;
    gather_idx_kernel<Td><<<grid_for(n < (1ll << 24) ? n : (1ll << 24)), kBlock, 0, s>>>(n, idx, src, dst);
}

__global__ void __launch_bounds__(1024) pair_reduce_kernel(int nblocks, const double *part, double *out) {
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
        a += part[2 * i];
        b += part[2 * i + 1];
    }
    a = block_sum(a);
    b = block_sum(b);
    if (threadIdx.x == 0) {
        out[0] = a;
        out[1] = b;
    }
}

// out[0], out[1] = sums of the (r^2, rhs^2) pairs written by the residual kernel.
void pair_reduce(int nblocks, const double *part, double *out, cudaStream_t s) {
    pair_reduce_kernel<<<1, 1024, 0, s>>>(nblocks, part, out);
}

// ---- block LU-SGS ----------------------------------------------------------
#define UCFD_BSW(B, CALL)                 \
    switch (B) {                          \
        case 1: { constexpr int BB = 1; CALL; break; } \
        case 2: { constexpr int BB = 2; CALL; break; } \
        case 4: { constexpr int BB = 4; CALL; break; } \
        case 5: { constexpr int BB = 5; CALL; break; } \
        default: ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "block size %d not built (1, 2, 4, 5)", B); \
    }

template <typename S>
void fs_blusgs_pack(int neles, int nvars, int B, long long N, double a0, const int *cell_ids,
                    const int *iperm, const double *rhs, const double *dt, S *rhs_s, double *rhs64,
                    double *D, cudaStream_t s) {
    if (neles <= 0) return;
    fs_blusgs_pack_kernel<S><<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, B, N, a0, cell_ids, iperm,
                                                                 rhs, dt, rhs_s, rhs64, D);
}

void fs_tblusgs_pack(int model, int neles, int nvars, int nt, long long N, double a0, double factor,
                     double betast, const int *cell_ids, const int *iperm, const double *uptsb,
                     const double *dsrc, const double *dt, double *D, cudaStream_t s) {
    if (neles <= 0) return;
    fs_tblusgs_pack_kernel<<<grid_for(neles), kBlock, 0, s>>>(model, neles, nvars, nt, N, a0, factor, betast,
                                                              cell_ids, iperm, uptsb, dsrc, dt, D);
}

template <typename S>
void fs_blusgs_prepare(int B, long long N, int P, long long nF, const int *nei, const int *slot,
                       const int8_t *side, const double *fa, const double *rv, const double *jmat,
                       const double *dd, double *D, double *LU64, S *LU_s, S *J_s, double *J64,
                       double *jt, cudaStream_t s) {
    if (N <= 0) return;
    const unsigned gt = (unsigned)((nF + 31) / 32);
    UCFD_BSW(B, (jmat_face_major_kernel<BB><<<gt, 256, 0, s>>>(nF, jmat, jt)));
    const int block = spread_block<double>(N, kPrepareThreads);
    UCFD_BSW(B, (fs_blusgs_prepare_kernel<S, BB><<<grid_for(N, block), block, 0, s>>>(
                    N, P, nei, slot, side, fa, rv, jt, dd, D, LU64, LU_s, J_s, J64)));
}

// Bulk-copy sweep: NST buffers per warp, 4 (NST 2) or 8 (NST 1) warps per
// block; grid capped at the blocks that fit on the device at once.
template <int B, int PW, int NST>
static void sweep_bulk_go(int t0, int t1, long long N, int var0, const int *nei, const float *fa,
                          const float *rv, const float *J, const float *LU, const float *rhs, float *du,
                          int *err, long long max_spin, const ::ucfd::SweepSplit<float> &sp, cudaStream_t s) {
    auto kern = fs_blusgs_sweep_bulk_kernel<B, PW, NST>;
    constexpr int threads = NST == 2 ? 128 : 256;
    constexpr int tiles_per_buf = kFold ? PW : PW + 1;  // J (and, in the exact build, LU) tiles
    constexpr size_t smem = (size_t)(threads / 32) * NST * (tiles_per_buf * B * B * 32 * sizeof(float) + 8);
    static int cap = 0;  // per instantiation: co-resident blocks on the device
    if (!cap) {
        UCFD_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0, dev = 0, sms = 0;
        UCFD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
        UCFD_CUDA(cudaGetDevice(&dev));
        UCFD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if (per_sm <= 0) ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "bulk-copy sweep kernel does not fit on the device");
        cap = per_sm * sms;
    }
    const long long tiles = (((long long)t1 + 31) >> 5) - (t0 >> 5);
    const long long want = (tiles + threads / 32 - 1) / (threads / 32);
    const unsigned g = (unsigned)(want < cap ? want : cap);
    kern<<<g, threads, smem, s>>>(t0, t1, N, var0, nei, fa, rv, J, LU, rhs, du, err, max_spin, sp);
}

// Unrolled sweep; in FP32 launched as a programmatic dependent of the
// previous level's launch (cudaLaunchAttributeProgrammaticStreamSerialization).
// In FP64 not: the waiting blocks crowd onto the SMs that run out of work
// first, and the FP64 pipe of those few SMs then bounds the level (226K cells,
// exact build: pair 510 us dependent, 389 us not; FMA 167 and 166 us; FP32
// 83 and 95 us).
template <typename S, int B, int PW>
static void sweep_dep_go(unsigned g, int block, cudaStream_t s, int t0, int t1, long long N, int P, int var0,
                         const int *nei, const S *fa, const S *rv, const S *J, const S *LU, const S *rhs, S *du,
                         const ::ucfd::SweepSplit<S> &sp) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    ::ucfd::SweepSplit<S> q = sp;
    if (std::is_same<S, double>::value) q.chained = 0;
    cfg.numAttrs = q.chained ? 1 : 0;
    UCFD_CUDA(cudaLaunchKernelEx(&cfg, fs_blusgs_sweep_kernel<S, B, PW>, t0, t1, N, P, var0, nei, fa, rv, J,
                                 LU, rhs, du, q));
}

// FP32 levels with at most this many cells take the register-hoisted kernel:
// they are bound by one thread's memory latency, not by bandwidth.
constexpr int kSmallLevel = 16384;

template <int B, int PW>
static void sweep_small_go(cudaStream_t s, int t0, int t1, long long N, int var0, const int *nei, const float *J,
                           const float *rhs, float *du, const ::ucfd::SweepSplit<float> &sp) {
    constexpr int threads = 128;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_for(t1 - (t0 & ~31), threads));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = sp.chained ? 1 : 0;
    UCFD_CUDA(cudaLaunchKernelEx(&cfg, fs_blusgs_sweep_small_kernel<B, PW>, t0, t1, N, var0, nei, J, rhs, du, sp));
}

// FP64 levels of at most this many cells take the kernel with B lanes per
// cell: a warp then holds 32 / B cells and costs about 60 FP64 instructions
// (fast build 32), against 270-420 (90) for 32 cells with one thread each.
// A lower + upper pair of two colours of hexahedra, 5x5, lanes / one thread
// per cell: 4000 cells a colour 23.6 / 56.9 us exact, 10.8 / 23.0 FMA; 7812
// 48.0 / 84.5, 15.9 / 29.3; 16384 87.6 / 101, 29.0 / 34.3; 23328 116 / 105,
// 32.9 / 37.8.  For these blocks the line could be at 16384; it is at half of
// that for the narrower ones, with fewer lanes per cell, not measured.
constexpr int kRowsCells = 8192;

template <int B, int PW>
static void sweep_rows_go(cudaStream_t s, int t0, int t1, long long N, int var0, const int *nei, const double *fv,
                          const double *J, const double *LU, const double *rhs, double *du,
                          const ::ucfd::SweepSplit<double> &sp) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid_for(t1 - t0, 32 / B));
    cfg.blockDim = dim3(32);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = sp.chained ? 1 : 0;
    UCFD_CUDA(cudaLaunchKernelEx(&cfg, fs_blusgs_sweep_rows_kernel<B, PW>, t0, t1, N, var0, nei, fv, J, LU, rhs, du,
                                 sp));
}

template <typename S>
void fs_blusgs_sweep(int B, int t0, int t1, long long N, int P, int var0, const int *nei, const S *fa,
                     const S *rv, const S *J, const S *LU, const S *rhs, S *du, int block,
                     int variant, int *err, long long max_spin, const ::ucfd::SweepSplit<S> &sp,
                     cudaStream_t s) {
    if (t1 <= t0) return;
    block = spread_block<S>(t1 - t0, block);
    // threads start at the tile boundary below t0 (see the kernel)
    const unsigned g = grid_for(t1 - (t0 & ~31), block);
    // variants 0 and 4: faces unrolled to the ELL width (6 or 4) when it
    // matches, each level a programmatic dependent launch of the previous;
    // variant 1: the face loop that stops at the first padding slot;
    // variants 2 / 3: FP32, ELL width 6 or 4, block 5: J and LU tiles staged
    // in shared memory by bulk copies, 2 / 1 buffers per warp.
    // All apply the faces in the same order with the same operations.
    if constexpr (std::is_same<S, double>::value) {
        // small levels, whatever the variant
        if (B > 1 && t1 - t0 <= kRowsCells && (P == 6 || P == 4)) {
            if (P == 6) {
                UCFD_BSW(B, (sweep_rows_go<BB, 6>(s, t0, t1, N, var0, nei, fa, J, LU, rhs, du, sp)));
            } else {
                UCFD_BSW(B, (sweep_rows_go<BB, 4>(s, t0, t1, N, var0, nei, fa, J, LU, rhs, du, sp)));
            }
            return;
        }
    }
    if constexpr (std::is_same<S, float>::value) {
        if ((variant == 2 || variant == 3) && B == 5 && (P == 6 || P == 4)) {
            if (!err) ::ucfd::fail(UCFD_ERR_ARGUMENT, "bulk-copy sweep needs an error flag");
            if (P == 6) {
                if (variant == 2) sweep_bulk_go<5, 6, 2>(t0, t1, N, var0, nei, fa, rv, J, LU, rhs, du, err, max_spin, sp, s);
                else sweep_bulk_go<5, 6, 1>(t0, t1, N, var0, nei, fa, rv, J, LU, rhs, du, err, max_spin, sp, s);
            } else {
                if (variant == 2) sweep_bulk_go<5, 4, 2>(t0, t1, N, var0, nei, fa, rv, J, LU, rhs, du, err, max_spin, sp, s);
                else sweep_bulk_go<5, 4, 1>(t0, t1, N, var0, nei, fa, rv, J, LU, rhs, du, err, max_spin, sp, s);
            }
            return;
        }
    }
    if (variant != 1 && (P == 6 || P == 4)) {
        if constexpr (std::is_same<S, float>::value) {
            if (kFold && B == 5 && t1 - t0 <= kSmallLevel) {
                if (P == 6) sweep_small_go<5, 6>(s, t0, t1, N, var0, nei, J, rhs, du, sp);
                else sweep_small_go<5, 4>(s, t0, t1, N, var0, nei, J, rhs, du, sp);
                return;
            }
        }
        if (P == 6) {
            UCFD_BSW(B, (sweep_dep_go<S, BB, 6>(g, block, s, t0, t1, N, P, var0, nei, fa, rv, J, LU, rhs, du, sp)));
        } else {
            UCFD_BSW(B, (sweep_dep_go<S, BB, 4>(g, block, s, t0, t1, N, P, var0, nei, fa, rv, J, LU, rhs, du, sp)));
        }
        return;
    }
    UCFD_BSW(B, (fs_blusgs_sweep_kernel<S, BB, 0><<<g, block, 0, s>>>(t0, t1, N, P, var0, nei, fa, rv, J, LU, rhs, du,
                                                                      sp)));
}

template <typename S>
void fs_blusgs_rhs_solve(int B, long long N, int var0, const S *LU, const S *b, S *c, cudaStream_t s) {
    if (N <= 0) return;
    UCFD_BSW(B, (fs_blusgs_rhs_solve_kernel<S, BB><<<grid_for(N), kBlock, 0, s>>>(N, var0, LU, b, c)));
}

template <typename Sx, typename R>
void fs_blusgs_residual(int B, long long N, int P, int var0, int nvars, const int *nei,
                        const double *fa, const double *rv, const double *J64, const double *D,
                        const double *rhs64, const Sx *x, R *r_out, double *part, int nblocks_max,
                        int *nblocks_used, cudaStream_t s) {
    const unsigned g = grid_for(N);
    if ((int)g > nblocks_max) ::ucfd::fail(UCFD_ERR_ARGUMENT, "residual partial buffer too small");
    *nblocks_used = (int)g;
    UCFD_BSW(B, (fs_blusgs_residual_kernel<Sx, R, BB><<<g, kBlock, 0, s>>>(
                    N, P, var0, nvars, nei, fa, rv, J64, D, rhs64, x, r_out, part)));
}

template <typename S>
void fs_blusgs_subres(int neles, int nvars, long long N, const int *cell_ids, const int *iperm,
                      const double *vol, const S *du, S *dup, double *res, cudaStream_t s) {
    if (neles <= 0) return;
    fs_blusgs_subres_kernel<S><<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, N, cell_ids, iperm, vol, du,
                                                                   dup, res);
}

template <typename S>
void fs_blusgs_update(int neles, int nvars, long long N, const int *cell_ids, const int *iperm,
                      const S *du, double *upts, cudaStream_t s) {
    if (neles <= 0) return;
    fs_blusgs_update_kernel<S><<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, N, cell_ids, iperm, du, upts);
}

// ---- Krylov ----------------------------------------------------------------
#define UCFD_KSW(B, CALL)                 \
    switch (B) {                          \
        case 1: { constexpr int BB = 1; CALL; break; } \
        case 2: { constexpr int BB = 2; CALL; break; } \
        case 3: { constexpr int BB = 3; CALL; break; } \
        case 4: { constexpr int BB = 4; CALL; break; } \
        case 5: { constexpr int BB = 5; CALL; break; } \
        case 6: { constexpr int BB = 6; CALL; break; } \
        case 7: { constexpr int BB = 7; CALL; break; } \
        default: ::ucfd::fail(UCFD_ERR_UNSUPPORTED, "block size %d not built (1..7)", B); \
    }

template <typename Tv, typename Ta>
void bsr_spmv(int B, int bn, int P, const int *col, const Tv *val, double alpha, const double *x,
              double beta, double *y, int block, cudaStream_t s) {
    if (bn <= 0) return;
    block = spread_block<Ta>(bn, block > 0 || sizeof(Ta) == 8 ? block : kBlock);
    const unsigned g = grid_for(bn, block);
    const int form = beta == 0.0 ? (alpha == 1.0 ? 1 : 3) : beta == 1.0 && alpha == -1.0 ? 2 : 0;
    // unrolled rows for the 5x5 systems (tets: diag + 4 faces; hexes: + 6);
    // FP32: vector loads of x where its base allows them (rows of 40 bytes)
    const bool vec = sizeof(Ta) == 4 && ((uintptr_t)x & 15) == 0;
#define UCFD_SPMV(BB, PW, VEC) \
    bsr_spmv_kernel<Tv, Ta, BB, PW, VEC><<<g, block, 0, s>>>(bn, P, col, val, alpha, x, beta, y, form)
    if (B == 5 && P <= 5) {
        if constexpr (sizeof(Ta) == 4) {
            if (vec) return UCFD_SPMV(5, 5, true);
        }
        UCFD_SPMV(5, 5, false);
        return;
    }
    if (B == 5 && P <= 7) {
        if constexpr (sizeof(Ta) == 4) {
            if (vec) return UCFD_SPMV(5, 7, true);
        }
        UCFD_SPMV(5, 7, false);
        return;
    }
    UCFD_KSW(B, (UCFD_SPMV(BB, 0, false)));
#undef UCFD_SPMV
}

template <typename Tl>
void pc_prepare(int B, int bn, const int *perm, const long long *dslot, const double *values,
                double *LU64, Tl *LU_l, int factor, cudaStream_t s) {
    if (bn <= 0) return;
    const int block = spread_block<double>(bn, 128);
    UCFD_KSW(B, (pc_prepare_kernel<Tl, BB><<<grid_for(bn, block), block, 0, s>>>(bn, perm, dslot, values, LU64,
                                                                             LU_l, factor)));
}

void ell_gather(int B, int bn, int P, const int *src, const double *vals, double *out64, float *out32,
                cudaStream_t s) {
    const long long warps = (long long)P * ((bn + 31) / 32);
    if (warps <= 0) return;
    UCFD_KSW(B, (ell_gather_kernel<BB><<<grid_for(warps, kGatherWarps<BB>), 32 * kGatherWarps<BB>, 0, s>>>(
                    bn, P, src, vals, out64, out32)));
}

void fingerprint(long long n, const int *a, unsigned long long *out, cudaStream_t s) {
    if (n <= 0) return;
    fingerprint_kernel<<<grid_for(n < (1ll << 22) ? n : (1ll << 22)), kBlock, 0, s>>>(n, a, out);
}

// Triangular steps, mode PC_BLUSGS / PC_BILU / PC_ILU (kernels_krylov.cuh).
// The working vector x has pc_stride entries per row.
template <typename T>
int pc_stride(int B) { return sizeof(T) == 4 && B > 3 ? 8 : B; }

template <typename T, int B, int PW, int MODE, bool LOWER>
static void pc_kernel_go(unsigned g, int block, cudaStream_t s, int t0, int t1, int bn, int P, const int *col,
                         const T *val, const T *LU, const int *perm, double *b, T *x) {
    constexpr int XS = sizeof(T) == 4 && B > 3 ? 8 : B;
    if constexpr (LOWER)
        pc_lower_kernel<T, B, PW, MODE, XS><<<g, block, 0, s>>>(t0, t1, bn, P, col, val, LU, perm, b, x);
    else
        pc_upper_kernel<T, B, PW, MODE, XS><<<g, block, 0, s>>>(t0, t1, bn, P, col, val, LU, perm, b, x);
}

template <typename T, int MODE, bool LOWER>
static void pc_step_go(int B, unsigned g, int block, cudaStream_t s, int t0, int t1, int bn, int P,
                       const int *col, const T *val, const T *LU, const int *perm, double *b, T *x) {
    if constexpr (MODE == PC_ILU) {
        if (B != 1) ::ucfd::fail(UCFD_ERR_ARGUMENT, "scalar ILU needs block size 1 (got %d)", B);
        pc_kernel_go<T, 1, 0, MODE, LOWER>(g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
        return;
    } else {
        if (B == 5 && P <= 6) {
            if (P <= 4) pc_kernel_go<T, 5, 4, MODE, LOWER>(g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
            else pc_kernel_go<T, 5, 6, MODE, LOWER>(g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
            return;
        }
        UCFD_KSW(B, (pc_kernel_go<T, BB, 0, MODE, LOWER>(g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x)));
    }
}

template <typename T, bool LOWER>
static void pc_step(int B, int t0, int t1, int bn, int P, const int *col, const T *val, const T *LU, const int *perm,
                    double *b, T *x, int block, int mode, cudaStream_t s) {
    if (t1 <= t0) return;
    block = spread_block<T>(t1 - t0, block > 0 || sizeof(T) == 8 ? block : kBlock);
    const unsigned g = grid_for(t1 - t0, block);
    if (mode == PC_BILU) pc_step_go<T, PC_BILU, LOWER>(B, g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
    else if (mode == PC_ILU) pc_step_go<T, PC_ILU, LOWER>(B, g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
    else pc_step_go<T, PC_BLUSGS, LOWER>(B, g, block, s, t0, t1, bn, P, col, val, LU, perm, b, x);
}

template <typename T>
void pc_lower(int B, int t0, int t1, int bn, int PL, const int *Lcol, const T *Lval, const T *LU, const int *perm,
              double *b, T *x, int block, int mode, cudaStream_t s) {
    pc_step<T, true>(B, t0, t1, bn, PL, Lcol, Lval, LU, perm, b, x, block, mode, s);
}

template <typename T>
void pc_upper(int B, int t0, int t1, int bn, int PU, const int *Ucol, const T *Uval, const T *LU, const int *perm,
              double *b, T *x, int block, int mode, cudaStream_t s) {
    pc_step<T, false>(B, t0, t1, bn, PU, Ucol, Uval, LU, perm, b, x, block, mode, s);
}

// One level of the ILU(0) factorisation (rows[t], t in [t0, t1)).
void ilu_factor(int B, int scalar, int t0, int t1, const int *rows, const int *rowptr, const int *colidx,
                const int *diagslots, double *vals, cudaStream_t s) {
    if (t1 <= t0) return;
    const int block = spread_block<double>(t1 - t0, 0);
    const unsigned g = grid_for(t1 - t0, block);
    if (scalar) {
        if (B != 1) ::ucfd::fail(UCFD_ERR_ARGUMENT, "scalar ILU needs block size 1 (got %d)", B);
        ilu_factor_scalar_kernel<true><<<g, block, 0, s>>>(t0, t1, rows, rowptr, colidx, diagslots, vals);
        return;
    }
    if (B > 1) {
        UCFD_KSW(B, (ilu_factor_rows_kernel<BB><<<grid_for(t1 - t0, 32 / BB), 32, 0, s>>>(t0, t1, rows, rowptr, colidx,
                                                                                         diagslots, vals)));
        return;
    }
    ilu_factor_scalar_kernel<false><<<g, block, 0, s>>>(t0, t1, rows, rowptr, colidx, diagslots, vals);
}

template <typename Ts, typename Td>
__global__ void convert_kernel(long long n, const Ts *src, Td *dst) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = convert_to<Td>(src[i]);
}

template <typename Ts, typename Td>
void convert(long long n, const Ts *src, Td *dst, cudaStream_t s) {
    if (n <= 0) return;
    convert_kernel<Ts, Td><<<grid_for(n < (1ll << 24) ? n : (1ll << 24)), kBlock, 0, s>>>(n, src, dst);
}

// dst = src where *flag is set.
__global__ void widen_if_kernel(long long n, const int *flag, const float *src, double *dst) {
    if (*flag == 0) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = to_double(src[i]);
}

void widen_if(long long n, const int *flag, const float *src, double *dst, cudaStream_t s) {
    if (n > 0) widen_if_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, flag, src, dst);
}

template <typename Ts>
__global__ void axpy_into_kernel(long long n, const Ts *x, double *y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] += to_double(x[i]);
}

template <typename Ts>
void axpy_into(long long n, const Ts *x, double *y, cudaStream_t s) {
    if (n <= 0) return;
    axpy_into_kernel<Ts><<<grid_for(n < (1ll << 24) ? n : (1ll << 24)), kBlock, 0, s>>>(n, x, y);
}

// y += x and out = ||x||_2 accumulated in FP64 (pseudo-time update).
template <typename S>
__global__ void axpy_norm_kernel(long long n, const S *x, S *y, double *part) {
    double t = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const S xv = x[i];
        y[i] += xv;
        t += (double)xv * (double)xv;
    }
    t = block_sum(t);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void __launch_bounds__(1024) sqrt_sum_kernel(int nb, const double *part, double *out) {
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) t += part[b];
    t = block_sum(t);
    if (threadIdx.x == 0) *out = sqrt(t);
}

// ---- GMRES pieces ----------------------------------------------------------
int gm_blocks(long long n) { return gm_grid(n); }

// gm_dots / gm_update: gm_launchers.cuh (their own translation unit, kern_gm.cu)

void gm_reduce(int nblocks, int K, const double *part, double *out, int accumulate, cudaStream_t s) {
    if (K <= 0) return;
    gm_reduce_kernel<<<K, kBlock, 0, s>>>(nblocks, part, out, accumulate);
}

void gm_sumsq(long long n, const double *x, double *part, cudaStream_t s) {
    gm_sumsq_kernel<<<gm_blocks(n), kBlock, 0, s>>>(n, x, part);
}

void gm_cycle_begin(int nblocks, const double *part, void *st, double *y, double *out_norm, cudaStream_t s) {
    gm_cycle_begin_kernel<<<1, kBlock, 0, s>>>(nblocks, part, (GmState *)st, y, out_norm);
}

void gm_scale(long long n, const void *st, const double *src, double *dst, cudaStream_t s) {
    gm_scale_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, (const GmState *)st, src, dst);
}

void gm_givens(int j, int ld, int nblocks, const double *part_norm, double *H, const double *h2, double *cs,
               double *sn, double *y, double haptol, double rel_floor, void *st, cudaStream_t s) {
    gm_givens_kernel<<<1, kBlock, 0, s>>>(j, ld, nblocks, part_norm, H, h2, cs, sn, y, haptol, rel_floor,
                                          (GmState *)st);
}

void gm_backsub(int ld, const double *H, double *y, const void *st, cudaStream_t s) {
    gm_backsub_kernel<<<1, 1, 0, s>>>(ld, H, y, (const GmState *)st);
}

void gm_solution(long long n, const double *V, long long ldv, const double *y, const void *st, double *x,
                 cudaStream_t s) {
    gm_solution_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, V, ldv, y, (const GmState *)st, x);
}

size_t gm_state_bytes() { return sizeof(GmState); }

template <typename S>
void axpy_norm(long long n, const S *x, S *y, double *part, double *out, cudaStream_t s) {
    const int nb = gm_blocks(n);
    axpy_norm_kernel<S><<<nb, kBlock, 0, s>>>(n, x, y, part);
    sqrt_sum_kernel<<<1, 1024, 0, s>>>(nb, part, out);
}

// The FP32 pseudo-time loop's state u += x, kept as a float-float pair: the
// working FP32 state hi (what the sweeps read) and a low part lo, together
// 48 significant bits, so an increment far below hi's rounding unit is kept
// in lo instead of being rounded away at every iteration.  The pair is
// updated by an error-free sum (Knuth's TwoSum of hi and x, the error added
// to lo) and renormalised (Dekker's Fast2Sum), all on the FP32 pipe: an FP64
// master would put four FP64 operations per value on GB300's narrow FP64
// pipe.  out = ||x||_2: each thread sums x^2 exactly split (x*x rounded plus
// its fma remainder) into a float-float accumulator, the thread sums are
// added in FP64.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}

__global__ void axpy_master_kernel(long long n, const float *x, float *hi, float *lo, double *part) {
    float ah = 0.f, al = 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float xv = x[i];
        float sh, se;
        two_sum(hi[i], xv, sh, se);
        const float t = lo[i] + se;
        const float nh = sh + t;
        hi[i] = nh;
        lo[i] = t - (nh - sh);
        const float p = __fmul_rn(xv, xv);
        const float pe = fmaf(xv, xv, -p);
        float qh, qe;
        two_sum(ah, p, qh, qe);
        const float ql = al + (qe + pe);
        ah = qh + ql;
        al = ql - (ah - qh);
    }
    double t = (double)ah + (double)al;
    t = block_sum(t);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

void axpy_master(long long n, const float *x, float *hi, float *lo, double *part, double *out, cudaStream_t s) {
    const int nb = gm_blocks(n);
    axpy_master_kernel<<<nb, kBlock, 0, s>>>(n, x, hi, lo, part);
    sqrt_sum_kernel<<<1, 1024, 0, s>>>(nb, part, out);
}

// Low part of the packed state (lusgs_pack's state, lusgs.c:8-37): with
// hi = (float)upts as fs_lusgs_pack rounds it, lo = (float)(upts - hi).
__global__ void state_lo_pack_kernel(int neles, int nvars, long long N, const int *cell_ids, const int *iperm,
                                     const double *upts, float *lo) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= neles) return;
    const long long k = iperm[cell_ids[idx]];
    for (int v = 0; v < nvars; ++v) {
        const double x = upts[idx + (long long)v * neles];
        lo[k + v * N] = (float)(x - (double)(float)x);
    }
}

void state_lo_pack(int neles, int nvars, long long N, const int *cell_ids, const int *iperm, const double *upts,
                   float *lo, cudaStream_t s) {
    if (neles <= 0) return;
    state_lo_pack_kernel<<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, N, cell_ids, iperm, upts, lo);
}

// rank_lusgs_update's write-back (lusgs.c:54-70) of the float-float state:
// upts = hi + lo in FP64.
__global__ void state_ff_update_kernel(int neles, int nvars, long long N, const int *cell_ids, const int *iperm,
                                       const float *hi, const float *lo, double *upts) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= neles) return;
    const long long k = iperm[cell_ids[idx]];
    for (int v = 0; v < nvars; ++v)
        upts[idx + (long long)v * neles] = (double)hi[k + v * N] + (double)lo[k + v * N];
}

void state_ff_update(int neles, int nvars, long long N, const int *cell_ids, const int *iperm, const float *hi,
                     const float *lo, double *upts, cudaStream_t s) {
    if (neles <= 0) return;
    state_ff_update_kernel<<<grid_for(neles), kBlock, 0, s>>>(neles, nvars, N, cell_ids, iperm, hi, lo, upts);
}

__global__ void __launch_bounds__(256) norm_finalize_kernel(int nblocks, const double *part, double *out) {
    const double t = block_sum_partials(part, nblocks, kMaxK);
    if (threadIdx.x == 0) *out = sqrt(t);
}

// out = ||x||_2 (two-pass, fixed order).
void norm2_to(long long n, const double *x, double *part, double *out, cudaStream_t s) {
    gm_sumsq_kernel<<<gm_blocks(n), kBlock, 0, s>>>(n, x, part);
    norm_finalize_kernel<<<1, kBlock, 0, s>>>(gm_blocks(n), part, out);
}

// ---- BiCGSTAB ----------------------------------------------------------------
size_t bc_state_bytes() { return sizeof(BcState); }

void bc_dot(long long n, const double *x, const double *y, double *part, const void *st, cudaStream_t s) {
    bc_dot_kernel<<<gm_blocks(n), kBlock, 0, s>>>(n, x, y, part, (const BcState *)st);
}
void bc_start(int nb, const double *part, void *st, int maxiter, cudaStream_t s) {
    bc_start_kernel<<<1, kBlock, 0, s>>>(nb, part, (BcState *)st, maxiter);
}
void bc_direction(long long n, const void *st, const double *r, const double *v, double *p, double *pt,
                  cudaStream_t s) {
    bc_direction_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, (const BcState *)st, r, v, p, pt);
}
void bc_alpha(int nb, const double *part, void *st, cudaStream_t s) {
    bc_alpha_kernel<<<1, kBlock, 0, s>>>(nb, part, (BcState *)st);
}
void bc_s(long long n, const void *st, const double *r, const double *v, double *sv, double *shat,
          cudaStream_t s) {
    bc_s_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, (const BcState *)st, r, v, sv, shat);
}
void bc_fused5(long long n, const double *rt, const double *sv, const double *t, double *part, const void *st,
               cudaStream_t s) {
    bc_fused5_kernel<<<gm_blocks(n), kBlock, 0, s>>>(n, rt, sv, t, part, (const BcState *)st);
}
void bc_omega(int nb, const double *part, void *st, double tol, double *hist, cudaStream_t s) {
    bc_omega_kernel<<<1, kBlock, 0, s>>>(nb, part, (BcState *)st, tol, hist);
}
void bc_update(long long n, const void *st, const double *pt, const double *shat, const double *sv,
               const double *t, double *x, double *r, cudaStream_t s) {
    bc_update_kernel<<<vec_grid(n), kBlock, 0, s>>>(n, (const BcState *)st, pt, shat, sv, t, x, r);
}
void bc_advance(void *st, int maxiter, cudaStream_t s) {
    bc_advance_kernel<<<1, 1, 0, s>>>((BcState *)st, maxiter);
}

}  // namespace UCFD_KNS
