// fftz.cu -- batched complex FFT along z (stride nx*ny), replacing the
// reference's nx*ny separate strided DFTI calls (Source/functions.cpp:
// 5858-5881, 6041-6046): forward unscaled, backward scaled 1/nz.
//
// One CTA owns TW consecutive z-columns (w = i + nx*j) and all nz rows.
// Loads and stores move whole rows of TW columns (coalesced, 512 B per warp
// for complex128).  The transform runs in shared memory as a mixed-radix
// Stockham sequence of passes (ping-pong buffers, natural order out): pass s
// with radix r and span p maps task i (k = i mod p) to
//     u_q = x[i + q*(n/r)] * w_{p r}^{q k},   U = DFT_r(u),
//     y[(i - k) r + k + q p] = U_q.
// Radices 2..8 are unrolled; any other prime factor uses a generic pass, and
// comes first, where no twiddles are needed (58 = 29 x 2, complex128: 49 us with
// one thread per butterfly).
#include <cuda_runtime.h>

#include "cplx.cuh"
#include "helm3d_internal.h"

namespace h3d {

struct FftK {
    int n, npass;
    int radix[kMaxPasses];
    int span[kMaxPasses];
    int twoff[kMaxPasses];
    int dftoff[kMaxPasses];
};

template <typename R, bool INV>
__device__ __forceinline__ cplx<R> tw_load(const cplx<R> *tw, int idx) {
    cplx<R> t = tw[idx];
    if (INV) t.y = -t.y;
    return t;
}

template <typename R, int RR, bool INV, int TW>
__device__ __forceinline__ void radix_task(const cplx<R> *__restrict__ src, cplx<R> *__restrict__ dst,
                                           const cplx<R> *__restrict__ tw, int twoff, int dftoff, int i,
                                           int m, int p, int col) {
    const int k = i % p;
    const int j = (i - k) * RR + k;
    cplx<R> u[RR];
#pragma unroll
    for (int q = 0; q < RR; q++) u[q] = src[(i + q * m) * TW + col];
    if (p > 1) {
#pragma unroll
        for (int q = 1; q < RR; q++) u[q] = cmul(u[q], tw_load<R, INV>(tw, twoff + k * RR + q));
    }
    cplx<R> U[RR];
    if (RR == 2) {
        U[0] = cadd(u[0], u[1]);
        U[1] = csub(u[0], u[1]);
    } else if (RR == 4) {
        cplx<R> a = cadd(u[0], u[2]), b = csub(u[0], u[2]);
        cplx<R> c = cadd(u[1], u[3]), d = csub(u[1], u[3]);
        // -i*d (forward) or +i*d (inverse)
        cplx<R> e = INV ? mkc<R>(-d.y, d.x) : mkc<R>(d.y, -d.x);
        U[0] = cadd(a, c);
        U[2] = csub(a, c);
        U[1] = cadd(b, e);
        U[3] = csub(b, e);
    } else {
#pragma unroll
        for (int q = 0; q < RR; q++) {
            cplx<R> acc = u[0];
#pragma unroll
            for (int t = 1; t < RR; t++) acc = cfma(u[t], tw_load<R, INV>(tw, dftoff + (q * t) % RR), acc);
            U[q] = acc;
        }
    }
#pragma unroll
    for (int q = 0; q < RR; q++) dst[(j + q * p) * TW + col] = U[q];
}

// A pass of any prime radix r: kGenQ outputs of one butterfly at a time per
// thread (the m butterflies of such a pass are too few to occupy the block one
// thread each), every input read once for them.
constexpr int kGenQ = 4;
template <typename R, bool INV, int TW>
__device__ void radix_pass_generic(const cplx<R> *__restrict__ src, cplx<R> *__restrict__ dst,
                                   const cplx<R> *__restrict__ tw, int twoff, int dftoff, int r, int m, int p,
                                   int col, int grp, int ngrp) {
    const int nq = (r + kGenQ - 1) / kGenQ;
    for (int e = grp; e < m * nq; e += ngrp) {
        const int i = e / nq, q0 = (e - i * nq) * kGenQ;
        const int k = i % p;
        const int j = (i - k) * r + k;
        cplx<R> acc[kGenQ];
        int idx[kGenQ], qs[kGenQ];   // (q t) mod r; past the last output: any q, not stored
#pragma unroll
        for (int u = 0; u < kGenQ; u++) {
            acc[u] = mkc<R>(0, 0);
            idx[u] = 0;
            qs[u] = q0 + u < r ? q0 + u : 0;
        }
        for (int t = 0; t < r; t++) {
            cplx<R> ut = src[(i + t * m) * TW + col];
            if (p > 1 && t > 0) ut = cmul(ut, tw_load<R, INV>(tw, twoff + k * r + t));
#pragma unroll
            for (int u = 0; u < kGenQ; u++) {
                acc[u] = cfma(ut, tw_load<R, INV>(tw, dftoff + idx[u]), acc[u]);
                idx[u] += qs[u];
                if (idx[u] >= r) idx[u] -= r;
            }
        }
#pragma unroll
        for (int u = 0; u < kGenQ; u++)
            if (q0 + u < r) dst[(j + (q0 + u) * p) * TW + col] = acc[u];
    }
}

template <typename R, int RR, bool INV, int TW>
__device__ __forceinline__ void radix_pass(const cplx<R> *__restrict__ src, cplx<R> *__restrict__ dst,
                                           const cplx<R> *__restrict__ tw, int to, int dof, int m, int p, int col,
                                           int grp, int ngrp) {
    for (int i = grp; i < m; i += ngrp) radix_task<R, RR, INV, TW>(src, dst, tw, to, dof, i, m, p, col);
}

template <typename R, bool INV, int TW>
__device__ cplx<R> *fft_passes(cplx<R> *A, cplx<R> *B, const FftK &fp, const cplx<R> *tw, int col, int grp,
                               int ngrp) {
    cplx<R> *src = A, *dst = B;
    for (int s = 0; s < fp.npass; s++) {
        const int r = fp.radix[s], p = fp.span[s], m = fp.n / r;
        const int to = fp.twoff[s], dof = fp.dftoff[s];
        switch (r) {
            case 2: radix_pass<R, 2, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            case 3: radix_pass<R, 3, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            case 4: radix_pass<R, 4, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            case 5: radix_pass<R, 5, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            case 7: radix_pass<R, 7, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            case 8: radix_pass<R, 8, INV, TW>(src, dst, tw, to, dof, m, p, col, grp, ngrp); break;
            default: radix_pass_generic<R, INV, TW>(src, dst, tw, to, dof, r, m, p, col, grp, ngrp); break;
        }
        __syncthreads();
        cplx<R> *t = src;
        src = dst;
        dst = t;
    }
    return src;
}

constexpr int kFftThreads = 256;
constexpr int kFftRows = 4;   // rows a thread loads at a time

// plane index of (row k, column w = i + nx*j) for right-hand side r
__device__ __forceinline__ long plane_index(const PlaneLayout &L, int r, int k, long w) {
    const long j = w / L.nx, i = w - j * L.nx;
    return (long)k * L.plane * L.R + (j * L.R + r) * L.nx + i;
}

template <typename R, int TW>
__global__ void __launch_bounds__(kFftThreads) fftz_forward_kernel(FftK fp, VecBatch x, double scale, ScaleBatch sc,
                                                                   cplx<R> *__restrict__ out, PlaneLayout L,
                                                                   const cplx<R> *__restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<R> *A = reinterpret_cast<cplx<R> *>(smem_raw);
    cplx<R> *B = A + (size_t)fp.n * TW;
    const int col = threadIdx.x % TW, grp = threadIdx.x / TW, ngrp = kFftThreads / TW;
    const int r = blockIdx.y;
    const long plane = L.plane;
    const double2 *xr = x.p + r * x.stride;
    const double s = scale * (sc.p ? sc.p[r * sc.stride] : 1.0);
    const long w = (long)blockIdx.x * TW + col;
    const bool valid = w < plane;
    for (int row0 = grp; row0 < fp.n; row0 += kFftRows * ngrp) {   // kFftRows loads in flight
        double2 v[kFftRows];
#pragma unroll
        for (int u = 0; u < kFftRows; u++) {
            const int row = row0 + u * ngrp;
            v[u] = valid && row < fp.n ? xr[(long)row * plane + w] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < kFftRows; u++) {
            const int row = row0 + u * ngrp;
            if (row < fp.n) A[row * TW + col] = cvt<cplx<R>, double2>(make_double2(v[u].x * s, v[u].y * s));
        }
    }
    __syncthreads();
    cplx<R> *res = fft_passes<R, false, TW>(A, B, fp, tw, col, grp, ngrp);
    if (!valid) return;
    const long obase = plane_index(L, r, 0, w), ostep = L.plane * L.R;
    for (int row = grp; row < fp.n; row += ngrp) out[obase + row * ostep] = res[row * TW + col];
}

template <typename R, int TW>
__global__ void __launch_bounds__(kFftThreads) fftz_inverse_kernel(FftK fp, const cplx<R> *__restrict__ in,
                                                                   PlaneLayout L, VecBatch y,
                                                                   const cplx<R> *__restrict__ tw, int mode,
                                                                   VecBatch wv, double scale, ScaleBatch sc,
                                                                   const double2 *__restrict__ dl) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<R> *A = reinterpret_cast<cplx<R> *>(smem_raw);
    cplx<R> *B = A + (size_t)fp.n * TW;
    const int col = threadIdx.x % TW, grp = threadIdx.x / TW, ngrp = kFftThreads / TW;
    const int r = blockIdx.y;
    const long plane = L.plane;
    const long w = (long)blockIdx.x * TW + col;
    const bool valid = w < plane;
    const long ibase = valid ? plane_index(L, r, 0, w) : 0, istep = L.plane * L.R;
    for (int row0 = grp; row0 < fp.n; row0 += kFftRows * ngrp) {
        cplx<R> v[kFftRows];
#pragma unroll
        for (int u = 0; u < kFftRows; u++) {
            const int row = row0 + u * ngrp;
            v[u] = valid && row < fp.n ? in[ibase + row * istep] : mkc<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < kFftRows; u++) {
            const int row = row0 + u * ngrp;
            if (row < fp.n) A[row * TW + col] = v[u];
        }
    }
    __syncthreads();
    cplx<R> *res = fft_passes<R, true, TW>(A, B, fp, tw, col, grp, ngrp);
    if (!valid) return;
    const double inv_n = 1.0 / (double)fp.n;
    double2 *yr = y.p + r * y.stride;
    const double2 *wr = mode == 1 ? wv.p + r * wv.stride : nullptr;
    const double s = scale * (sc.p ? sc.p[r * sc.stride] : 1.0);
    for (int row = grp; row < fp.n; row += ngrp) {
        const long idx = (long)row * plane + w;
        double2 t = cvt<double2, cplx<R>>(res[row * TW + col]);
        t.x *= inv_n;
        t.y *= inv_n;
        if (mode == 1) {
            const double2 a = wr[idx], d = dl[idx];
            t = make_double2(s * a.x - (d.x * t.x - d.y * t.y), s * a.y - (d.x * t.y + d.y * t.x));
        }
        if (y.c64) reinterpret_cast<float2 *>(y.p)[r * y.stride + idx] = cvt<float2, double2>(t);
        else yr[idx] = t;
    }
}

static FftK to_k(const FftPlan &p) {
    FftK k;
    k.n = p.n;
    k.npass = p.npass;
    for (int s = 0; s < kMaxPasses; s++) {
        k.radix[s] = p.radix[s];
        k.span[s] = p.span[s];
        k.twoff[s] = p.twoff[s];
        k.dftoff[s] = p.dftoff[s];
    }
    return k;
}

// Columns per CTA: 32, or 16 (256-byte rows in complex128, still whole
// sectors) where 32 would leave less than two CTAs per SM or do not fit the
// shared memory (two buffers of n x TW elements).
template <typename R> static int pick_tw(int n, const PlaneLayout &L) {
    const size_t cap = device_info().smem_optin;
    const bool few = ((L.plane + 31) / 32) * L.R < 2L * device_info().sm_count;
    if (!few && (size_t)2 * n * 32 * sizeof(cplx<R>) <= cap) return 32;
    if ((size_t)2 * n * 16 * sizeof(cplx<R>) <= cap) return 16;
    return 0;
}

template <typename R, int TW>
static int fwd_impl(const VecBatch &x, double scale, const ScaleBatch &sc, void *planes, const PlaneLayout &L,
                    const FftPlan &plan, const void *tw, cudaStream_t s) {
    size_t smem = (size_t)2 * plan.n * TW * sizeof(cplx<R>);
    auto kern = fftz_forward_kernel<R, TW>;
    if (!smem_limit_max(kern, smem))
        return HELM3D_ERR_CUDA;
    dim3 grid((unsigned)((L.plane + TW - 1) / TW), (unsigned)L.R);
    kern<<<grid, kFftThreads, smem, s>>>(to_k(plan), x, scale, sc, (cplx<R> *)planes, L, (const cplx<R> *)tw);
    return cudaGetLastError() == cudaSuccess ? HELM3D_OK : HELM3D_ERR_CUDA;
}

template <typename R, int TW>
static int inv_impl(const void *planes, const PlaneLayout &L, const VecBatch &y, const FftPlan &plan, const void *tw,
                    int mode, const VecBatch &w, double scale, const ScaleBatch &sc, const double2 *dl,
                    cudaStream_t s) {
    size_t smem = (size_t)2 * plan.n * TW * sizeof(cplx<R>);
    auto kern = fftz_inverse_kernel<R, TW>;
    if (!smem_limit_max(kern, smem))
        return HELM3D_ERR_CUDA;
    dim3 grid((unsigned)((L.plane + TW - 1) / TW), (unsigned)L.R);
    kern<<<grid, kFftThreads, smem, s>>>(to_k(plan), (const cplx<R> *)planes, L, y, (const cplx<R> *)tw, mode, w,
                                         scale, sc, dl);
    return cudaGetLastError() == cudaSuccess ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_fft_forward(bool c64, const VecBatch &x, double scale, const ScaleBatch &sc, void *planes,
                       const PlaneLayout &L, const FftPlan &plan, const void *tw, cudaStream_t s) {
    if (c64) {
        int tw_ = pick_tw<float>(plan.n, L);
        if (tw_ == 32) return fwd_impl<float, 32>(x, scale, sc, planes, L, plan, tw, s);
        if (tw_ == 16) return fwd_impl<float, 16>(x, scale, sc, planes, L, plan, tw, s);
    } else {
        int tw_ = pick_tw<double>(plan.n, L);
        if (tw_ == 32) return fwd_impl<double, 32>(x, scale, sc, planes, L, plan, tw, s);
        if (tw_ == 16) return fwd_impl<double, 16>(x, scale, sc, planes, L, plan, tw, s);
    }
    return HELM3D_ERR_ARG;
}

int launch_fft_inverse(bool c64, const void *planes, const PlaneLayout &L, const VecBatch &y, const FftPlan &plan,
                       const void *tw, int mode, const VecBatch &w, double scale, const ScaleBatch &sc,
                       const double2 *dl, cudaStream_t s) {
    if (c64) {
        int tw_ = pick_tw<float>(plan.n, L);
        if (tw_ == 32) return inv_impl<float, 32>(planes, L, y, plan, tw, mode, w, scale, sc, dl, s);
        if (tw_ == 16) return inv_impl<float, 16>(planes, L, y, plan, tw, mode, w, scale, sc, dl, s);
    } else {
        int tw_ = pick_tw<double>(plan.n, L);
        if (tw_ == 32) return inv_impl<double, 32>(planes, L, y, plan, tw, mode, w, scale, sc, dl, s);
        if (tw_ == 16) return inv_impl<double, 16>(planes, L, y, plan, tw, mode, w, scale, sc, dl, s);
    }
    return HELM3D_ERR_ARG;
}

}  // namespace h3d
