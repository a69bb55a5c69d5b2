// ztrans.cu -- dense transform along z with the eigenvectors of the z
// operator with its PML (the HELM3D_ZT_PML_EIGEN preconditioner):
//   forward  planes[k][w] = sum_j Wi[k][j] (scale x[j][w])   (complex128 in, P out)
//   inverse  y[k][w]      = sum_j W[k][j] planes[j][w]        (P in, complex128 out)
// for every z-column w = i + nx*j of the grid, in FP64 whatever the plane
// precision (W is far from unitary: cond(W) ~ 1e4 for 12-point PMLs at
// nz = 128).  One CTA owns 16 consecutive columns: their nz x 16 input tile is
// staged in shared memory with coalesced row loads; a thread accumulates KR
// output rows of one column over j, the matrix staged KC columns at a time in
// shared memory (transposed: the rows of one j are adjacent), the next KC in
// registers meanwhile.  Bound by the FP64 pipe (4 nz FMAs per output): with the
// matrix read through L1 entry by entry and 32 columns per CTA, fewer CTAs
// than SMs, a transform of 57 x 48 x 53 took 42 us.
#include <cuda_runtime.h>

#include "cplx.cuh"
#include "helm3d_internal.h"

namespace h3d {

constexpr int kZtCols = 16, kZtThreads = 256, kZtGroups = kZtThreads / kZtCols;
constexpr int kZtKC = 8;   // matrix columns per stage

// plane index of (row k, column w = i + nx*j) for right-hand side r
__device__ __forceinline__ long zt_plane_index(const PlaneLayout &L, int r, int k, long w) {
    const long j = w / L.nx, i = w - j * L.nx;
    return (long)k * L.plane * L.R + (j * L.R + r) * L.nx + i;
}

// KR: output rows per thread; a pass over j covers kZtGroups * KR rows
template <typename R, bool FWD, int KR>
__global__ void __launch_bounds__(kZtThreads) ztrans_kernel(PlaneLayout L, VecBatch vec, double scale, ScaleBatch sc,
                                                            cplx<R> *__restrict__ planes,
                                                            const double2 *__restrict__ M) {
    typedef cplx<R> Cx;
    constexpr int KB = kZtGroups * KR;   // rows per pass
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *tile = reinterpret_cast<double2 *>(smem_raw);   // [nz][kZtCols]
    double2 *ms = tile + (size_t)L.nz * kZtCols;             // [kZtKC][KB]
    const int nz = L.nz;
    const long plane = L.plane;
    const int col = threadIdx.x % kZtCols, grp = threadIdx.x / kZtCols;
    const int r = blockIdx.y;
    double2 *v_r = vec.p + r * vec.stride;
    const double s = scale * (sc.p ? sc.p[r * sc.stride] : 1.0);
    const long w = (long)blockIdx.x * kZtCols + col;
    const bool valid = w < plane;
    const long pbase = valid ? zt_plane_index(L, r, 0, w) : 0, pstep = plane * L.R;
    for (int j0 = grp; j0 < nz; j0 += 4 * kZtGroups) {   // 4 loads in flight
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int j = j0 + u * kZtGroups;
            v[u] = make_double2(0, 0);
            if (valid && j < nz) {
                if (FWD) {
                    const double2 x = v_r[(long)j * plane + w];
                    v[u] = make_double2(s * x.x, s * x.y);
                } else {
                    v[u] = cvt<double2, Cx>(planes[pbase + j * pstep]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (j0 + u * kZtGroups < nz) tile[(j0 + u * kZtGroups) * kZtCols + col] = v[u];
    }
    for (int k0 = 0; k0 < nz; k0 += KB) {
        double2 acc[KR];
#pragma unroll
        for (int q = 0; q < KR; q++) acc[q] = make_double2(0, 0);
        // stage entries e = (row e / kZtKC, column e % kZtKC): coalesced runs of kZtKC
        constexpr int PER = (KB * kZtKC + kZtThreads - 1) / kZtThreads;
        double2 nx[PER];
        auto fetch = [&](int j0) {
#pragma unroll
            for (int u = 0; u < PER; u++) {
                const int e = threadIdx.x + u * kZtThreads, k = k0 + e / kZtKC, j = j0 + e % kZtKC;
                nx[u] = e < KB * kZtKC && k < nz && j < nz ? __ldg(&M[(long)k * nz + j]) : make_double2(0, 0);
            }
        };
        fetch(0);
        for (int j0 = 0; j0 < nz; j0 += kZtKC) {
            __syncthreads();   // the tile is in (first), the last stage read
#pragma unroll
            for (int u = 0; u < PER; u++) {
                const int e = threadIdx.x + u * kZtThreads;
                if (e < KB * kZtKC) ms[(e % kZtKC) * KB + e / kZtKC] = nx[u];
            }
            __syncthreads();
            if (j0 + kZtKC < nz) fetch(j0 + kZtKC);
            const int jn = min(kZtKC, nz - j0);
            for (int j = 0; j < jn; j++) {
                const double2 t = tile[(j0 + j) * kZtCols + col];
                const double2 *m = ms + j * KB + grp * KR;
#pragma unroll
                for (int q = 0; q < KR; q++) acc[q] = cfma(m[q], t, acc[q]);
            }
        }
        if (valid) {
#pragma unroll
            for (int q = 0; q < KR; q++) {
                const int k = k0 + grp * KR + q;
                if (k >= nz) break;
                if (FWD) planes[pbase + k * pstep] = cvt<Cx, double2>(acc[q]);
                else if (vec.c64) reinterpret_cast<float2 *>(vec.p)[r * vec.stride + (long)k * plane + w] = cvt<float2, double2>(acc[q]);
                else v_r[(long)k * plane + w] = acc[q];
            }
        }
    }
}

template <typename R, bool FWD, int KR>
static int zt_go(const PlaneLayout &L, const VecBatch &vec, double scale, const ScaleBatch &sc, void *planes,
                 const double2 *M, cudaStream_t s) {
    const size_t smem = ((size_t)L.nz * kZtCols + kZtKC * kZtGroups * KR) * sizeof(double2);
    auto kern = ztrans_kernel<R, FWD, KR>;
    if (smem > device_info().smem_optin) return HELM3D_ERR_ARG;
    if (!smem_limit_max(kern, smem)) return HELM3D_ERR_CUDA;
    const dim3 grid((unsigned)((L.plane + kZtCols - 1) / kZtCols), (unsigned)L.R);
    kern<<<grid, kZtThreads, smem, s>>>(L, vec, scale, sc, (cplx<R> *)planes, M);
    return cudaGetLastError() == cudaSuccess ? HELM3D_OK : HELM3D_ERR_CUDA;
}

// rows per thread: enough for one pass over j up to nz = 128
template <typename R, bool FWD>
static int zt_impl(const PlaneLayout &L, const VecBatch &vec, double scale, const ScaleBatch &sc, void *planes,
                   const double2 *M, cudaStream_t s) {
    if ((size_t)L.nz * 32 * sizeof(double2) > device_info().smem_optin) return HELM3D_ERR_ARG;   // nz > 454
    if (L.nz <= 2 * kZtGroups) return zt_go<R, FWD, 2>(L, vec, scale, sc, planes, M, s);
    if (L.nz <= 4 * kZtGroups) return zt_go<R, FWD, 4>(L, vec, scale, sc, planes, M, s);
    return zt_go<R, FWD, 8>(L, vec, scale, sc, planes, M, s);
}

int launch_ztrans_forward(bool c64, const VecBatch &x, double scale, const ScaleBatch &sc, void *planes,
                          const PlaneLayout &L, const double2 *Wi, cudaStream_t s) {
    return c64 ? zt_impl<float, true>(L, x, scale, sc, planes, Wi, s)
               : zt_impl<double, true>(L, x, scale, sc, planes, Wi, s);
}

int launch_ztrans_inverse(bool c64, const void *planes, const PlaneLayout &L, const VecBatch &y, const double2 *W,
                          cudaStream_t s) {
    const ScaleBatch none = {nullptr, 0};
    return c64 ? zt_impl<float, false>(L, y, 1.0, none, (void *)planes, W, s)
               : zt_impl<double, false>(L, y, 1.0, none, (void *)planes, W, s);
}

}  // namespace h3d
