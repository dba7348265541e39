// kernels_adjoint.cuh -- reverse-mode derivative of one colored LU-SGS step
// (array layout), as transposed sweeps.
//
// Forward (lusgs.c:87-257 on the colour-renumbered mesh):
//   D_i    = 1/(dt_i f) + 1/2 sum_f lam_fi s_fi
//   lower  dQ*_i = (R_i - 1/2 sum_{f in L(i)} G_fi(dQ*_j)) / D_i
//   upper  dQ_i  = dQ*_i - 1/2 D_i^-1 sum_{f in U(i)} G_fi(dQ_j)
//   G_fi(d) = [F(u_j + d; n_fi) - F(u_j; n_fi) - lam_fi d] s_fi
// Reverse: first the upper sweep transposed (colours ascending), then the
// lower sweep transposed (colours descending), then the diagonal.  Each
// thread owns one cell and *pulls* the contributions of the neighbours
// that used it (through the reverse-face map rface), so no atomics are
// needed and every output element has one writer.
#pragma once

#include "kernels_common.cuh"
#include "kargs.h"

namespace UCFD_KNS {

// J = dF(w; n)/dw of the Euler flux (flux.c:29-67) at one state w, including
// the branch where the pressure floor replaces the energy: what J^T v needs
// of w for any normal n and vector v.
//   v . F = v0 th + (v_m.m + vE H) c + (v_m.n) p,  th = m.n, c = th / rho,
//   H = Ee + p, so with G = (v_m.m + vE H) / rho, A = vE c, B = v_m.n
//   d/drho = -G c + A dH/drho + B dp/drho
//   d/dm_d = n_d (v0 + G) + v_d c + m_d (A hm + B pm),  dH/dm_d = hm m_d, dp/dm_d = pm m_d
//   d/dE   = A dH/dE + B dp/dE
// About 30 multiply-adds per face instead of 60 with J formed entry by entry;
// the derivatives of p and H are formed once per cell.
template <typename T, int NFV, int NDIMS>
struct FluxJt {
    T m[NDIMS], ir, H, pr, hr, pm, hm, pe, he;

    __device__ __forceinline__ FluxJt(T gamma, T pmin, const T *w) {
        T q = T(0);
#pragma unroll
        for (int d = 0; d < NDIMS; ++d) {
            m[d] = w[d + 1];
            q += m[d] * m[d];
        }
        ir = T(1) / w[0];
        const T gm1 = gamma - T(1), E = w[NFV - 1];
        const T ke = T(0.5) * q * ir;
        const T kr = ke * ir;  // -d(ke)/drho
        const T p = gm1 * (E - ke);
        if (p < pmin) {  // p = pmin, Ee = pmin / (gamma - 1) + ke
            H = pmin / gm1 + ke + pmin;
            pr = pm = pe = he = T(0);
            hr = -kr;
            hm = ir;
        } else {
            H = E + p;
            pr = hr = gm1 * kr;
            pm = hm = -gm1 * ir;
            pe = gm1;
            he = T(1) + gm1;
        }
    }

    // out = J^T v
    __device__ __forceinline__ void apply(const T *n, const T *v, T *out) const {
        T th = T(0), vm = T(0), B = T(0);
#pragma unroll
        for (int d = 0; d < NDIMS; ++d) {
            th += m[d] * n[d];
            vm += v[d + 1] * m[d];
            B += v[d + 1] * n[d];
        }
        const T c = th * ir, G = (vm + v[NFV - 1] * H) * ir, A = v[NFV - 1] * c;
        out[0] = A * hr + B * pr - G * c;
        const T vG = v[0] + G, tm = A * hm + B * pm;
#pragma unroll
        for (int d = 0; d < NDIMS; ++d) out[d + 1] = n[d] * vG + v[d + 1] * c + m[d] * tm;
        out[NFV - 1] = A * he + B * pe;
    }
};

using AdjArgs = ::ucfd::AdjArgs;

// A cell's neighbours, their side of this sweep and the reverse faces, all
// requested before anything depends on them, six faces f0 .. f0 + 5 at a time
// (a hexahedron's; wider rows take several): bit f of lo / hi set where the
// neighbour of face f0 + f has a lower / higher colour.  Walked face by face
// these were four dependent loads per face.
struct AdjFaces {
    static constexpr int NB = 6;
    int nb[NB], rf[NB];
    unsigned lo = 0u, hi = 0u;

    __device__ __forceinline__ AdjFaces(const AdjArgs &a, int i, int ci, int f0) {
        const long long N = a.neles;
#pragma unroll
        for (int f = 0; f < NB; ++f) {
            nb[f] = f0 + f < a.nface ? __ldg(a.nei + (f0 + f) * N + i) : i;
            rf[f] = f0 + f < a.nface ? __ldg(a.rface + (f0 + f) * N + i) : 0;
        }
        int lc[NB];
#pragma unroll
        for (int f = 0; f < NB; ++f) lc[f] = nb[f] != i ? __ldg(a.lcolor + nb[f]) : ci;
#pragma unroll
        for (int f = 0; f < NB; ++f) {
            lo |= lc[f] < ci ? 1u << f : 0u;
            hi |= lc[f] > ci ? 1u << f : 0u;
        }
    }
    __device__ __forceinline__ void pick(int f, int &k, int &fp) const {
        k = nb[0];
        fp = rf[0];
#pragma unroll
        for (int q = 1; q < NB; ++q) {
            k = f == q ? nb[q] : k;
            fp = f == q ? rf[q] : fp;
        }
    }
};

// acc += s (J^T w - lam w) for every face of the mask, through which the cell
// is a neighbour's neighbour: w [NFV][N] of that neighbour k, s, lam and the
// normal of k's own face fp.
template <typename T, int NFV, int NDIMS>
__device__ __forceinline__ void adj_pull(const AdjArgs &a, const AdjFaces &F, unsigned mask,
                                         const FluxJt<T, NFV, NDIMS> &J, const T *fnv, const T *vec, const T *fspr,
                                         const T *wsrc, T *acc) {
    const long long N = a.neles;
#pragma unroll 1
    while (mask) {
        int k, fp;
        F.pick(__ffs(mask) - 1, k, fp);
        mask &= mask - 1u;
        T w[NFV], n[NDIMS], y[NFV];
#pragma unroll
        for (int v = 0; v < NFV; ++v) w[v] = wsrc[v * N + k];
#pragma unroll
        for (int d = 0; d < NDIMS; ++d) n[d] = __ldg(vec + (fp * NDIMS + d) * N + k);
        const T s = __ldg(fnv + fp * N + k), lam = __ldg(fspr + fp * N + k);
        J.apply(n, w, y);
#pragma unroll
        for (int v = 0; v < NFV; ++v) acc[v] += s * (y[v] - lam * w[v]);
    }
}

// Transposed upper sweep for one colour.  qbar = adjoint of dQ (final for
// this cell once its lower-coloured neighbours are done), dbar = adjoint of
// D (upper part), gfspr initialised for every face of the cell.  wbuf holds
// -qbar / (2 D) of the cells already processed, what their neighbours pull,
// so a face costs no division (FP64 division is a long sequence on GB300's
// FP64 pipe).  Gradients of a 64^3-cell step in FP64, forward and backward:
// 2.17 -> 1.69 ms with the transposed sweeps in this form (before, faces one
// after the other, J entry by entry and a division per face).
template <typename T, int NFV, int NDIMS>
__global__ void __launch_bounds__(256) adj_upper_kernel(AdjArgs a, T gamma, T pmin, const T *fnv, const T *vec,
                                                        const T *fspr, const T *upts, const T *diag, const T *dub,
                                                        const T *dq, const T *gdq, T *qbar, T *wbuf, T *dbar,
                                                        T *gfspr) {
    const int t = a.t0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.t1) return;
    const long long N = a.neles;
    const int i = __ldg(a.icolor + t);
    const int ci = __ldg(a.lcolor + i);
    AdjFaces F(a, i, ci, 0);
    T qb[NFV], st[NFV], dqi[NFV], dui[NFV];
#pragma unroll
    for (int v = 0; v < NFV; ++v) {
        qb[v] = gdq[v * N + i];
        dqi[v] = dq[v * N + i];
        dui[v] = dub[v * N + i];
        st[v] = upts[v * N + i] + dqi[v];  // state u_i + dQ_i
    }
    const T iD = T(1) / diag[i];
    const FluxJt<T, NFV, NDIMS> J(gamma, pmin, st);
    adj_pull(a, F, F.lo, J, fnv, vec, fspr, wbuf, qb);
#pragma unroll 1
    for (int f0 = AdjFaces::NB; f0 < a.nface; f0 += AdjFaces::NB) {
        F = AdjFaces(a, i, ci, f0);
        adj_pull(a, F, F.lo, J, fnv, vec, fspr, wbuf, qb);
    }
    T db = T(0);
#pragma unroll
    for (int v = 0; v < NFV; ++v) {
        qbar[v * N + i] = qb[v];
        wbuf[v * N + i] = T(-0.5) * iD * qb[v];
        db -= qb[v] * (dqi[v] - dui[v]);
    }
    dbar[i] = db * iD;
    if (a.nface > AdjFaces::NB) F = AdjFaces(a, i, ci, 0);
#pragma unroll 1
    for (int f = 0, f6 = 0; f < a.nface; ++f, ++f6) {
        if (f6 == AdjFaces::NB) {
            F = AdjFaces(a, i, ci, f);
            f6 = 0;
        }
        T g = T(0);
        if ((F.hi >> f6) & 1u) {
            int j, fp;
            F.pick(f6, j, fp);
            T dot = T(0);
#pragma unroll
            for (int v = 0; v < NFV; ++v) dot += __ldg(dq + v * N + j) * qb[v];
            g = T(0.5) * __ldg(fnv + f * N + i) * iD * dot;
        }
        gfspr[f * N + i] = g;
    }
}

// Transposed lower sweep for one colour, then the diagonal: grhs, gdt and
// the rest of gfspr.  wbuf = qstar / D of the cells already processed.
template <typename T, int NFV, int NDIMS>
__global__ void __launch_bounds__(256) adj_lower_kernel(AdjArgs a, T gamma, T pmin, T factor, const T *fnv,
                                                        const T *vec, const T *fspr, const T *dt, const T *upts,
                                                        const T *diag, const T *dub, const T *qbar, T *wbuf,
                                                        const T *dbar, T *grhs, T *gdt, T *gfspr) {
    const int t = a.t0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.t1) return;
    const long long N = a.neles;
    const int i = __ldg(a.icolor + t);
    const int ci = __ldg(a.lcolor + i);
    AdjFaces F(a, i, ci, 0);
    T qs[NFV], st[NFV], dui[NFV], acc[NFV];
#pragma unroll
    for (int v = 0; v < NFV; ++v) {
        qs[v] = qbar[v * N + i];
        dui[v] = dub[v * N + i];
        st[v] = upts[v * N + i] + dui[v];  // state u_i + dQ*_i
        acc[v] = T(0);
    }
    const T iD = T(1) / diag[i];
    const FluxJt<T, NFV, NDIMS> J(gamma, pmin, st);
    adj_pull(a, F, F.hi, J, fnv, vec, fspr, wbuf, acc);
#pragma unroll 1
    for (int f0 = AdjFaces::NB; f0 < a.nface; f0 += AdjFaces::NB) {
        F = AdjFaces(a, i, ci, f0);
        adj_pull(a, F, F.hi, J, fnv, vec, fspr, wbuf, acc);
    }
    T wi[NFV];
    T db = dbar[i];
#pragma unroll
    for (int v = 0; v < NFV; ++v) {
        wi[v] = (qs[v] - T(0.5) * acc[v]) * iD;
        wbuf[v * N + i] = wi[v];
        grhs[v * N + i] = wi[v];
        db -= wi[v] * dui[v];
    }
    // D_i = 1/(dt_i f) + 1/2 sum_f lam_fi s_fi
    const T dti = dt[i];
    gdt[i] = -db / (dti * dti * factor);
    const T hdb = T(0.5) * db;
    if (a.nface > AdjFaces::NB) F = AdjFaces(a, i, ci, 0);
#pragma unroll 1
    for (int f = 0, f6 = 0; f < a.nface; ++f, ++f6) {
        if (f6 == AdjFaces::NB) {
            F = AdjFaces(a, i, ci, f);
            f6 = 0;
        }
        const T s = __ldg(fnv + f * N + i);
        T g = gfspr[f * N + i] + s * hdb;
        if ((F.lo >> f6) & 1u) {
            int j, fp;
            F.pick(f6, j, fp);
            T dot = T(0);
#pragma unroll
            for (int v = 0; v < NFV; ++v) dot += __ldg(dub + v * N + j) * wi[v];
            g += T(0.5) * s * dot;
        }
        gfspr[f * N + i] = g;
    }
}

}  // namespace UCFD_KNS
