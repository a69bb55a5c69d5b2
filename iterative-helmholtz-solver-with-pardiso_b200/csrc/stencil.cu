// stencil.cu -- the complex 7-point PML-stretched operator (mode N) and its
// conjugate transpose, complex128:
//   (A u)_ijk = sum_a [cp_a (u_{+a} - u) + cm_a (u_{-a} - u)]
//               + omega^2 s2_ijk (1 + i beta) u_ijk,        u = 0 off the grid
// with cp_a(i) = alpha(i) alpha(i+1/2)/h^2 and cm_a(i) = alpha(i) alpha(i-1/2)/h^2
// (the reference's 5-point form, beta2D_pml, Source/functions.cpp:2347-2402,
// carried to z).  Bound by HBM (40 bytes a point), so every load of a CTA's
// points is issued before the first use; a kernel that marched along z with one
// plane's loads in flight, or three in a ring of shared-memory planes, reached
// 37-46 % of it.  stencil_block_kernel: a CTA owns 32 x 8 x ZB points, copies
// them with their halo into shared memory at once (asynchronous copies,
// zero-filled off the grid, which is the operator's u = 0 there), s2 into
// registers meanwhile, and goes through the ZB planes from shared memory, the z
// neighbours in registers, f (a residual's) read as its plane comes.  stencil_kernel: the same from registers and L1
// without a barrier, a thread per ZB points of a column, for grids too small to
// fill the SMs with such blocks.  The grid's z dimension enumerates (source, z
// block) pairs, source-major or source-minor (autotuned, with ZB).  The input x
// is complex128, or complex64 (TX = float2: FGMRES's Z basis of a complex64
// preconditioner), widened to complex128 as it is read; the arithmetic and y
// are complex128.
#include <cuda_runtime.h>

#include "cplx.cuh"
#include "helm3d_internal.h"
#include "ptx.cuh"

namespace h3d {

constexpr int kStX = 32, kStY = 8;

template <bool ADJ, typename TX, int ZB>
__global__ void __launch_bounds__(kStX *kStY) stencil_kernel(StencilArgs a) {
    const int i = blockIdx.x * kStX + threadIdx.x;
    const int j = blockIdx.y * kStY + threadIdx.y;
    if (i >= a.nx || j >= a.ny) return;
    const int nzc = (a.nz + ZB - 1) / ZB;
    // source-minor order: the R sources of a z block are adjacent in launch
    // order and run together, so their reads of s2 and the coefficient
    // tables meet in L2 instead of coming from DRAM once per source
    const int r = a.src_fast ? (int)(blockIdx.z % a.R) : (int)(blockIdx.z / nzc);
    const int zc = a.src_fast ? (int)(blockIdx.z / a.R) : (int)(blockIdx.z - r * nzc);
    const int k0 = zc * ZB;
    const long plane = (long)a.nx * a.ny;
    const long idx0 = (long)k0 * plane + (long)j * a.nx + i;
    const TX *x = reinterpret_cast<const TX *>(a.x.p) + r * a.x.stride + idx0;
    double2 *yout = a.y.p + r * a.y.stride + idx0;
    const double2 *fin = a.f.p ? a.f.p + r * a.f.stride + idx0 : nullptr;
    const double *s2 = a.s2 + idx0;
    const bool hxm = i > 0, hxp = i + 1 < a.nx, hym = j > 0, hyp = j + 1 < a.ny;

    // ---- loads: u[q] = x at k0 - 1 + q, nb[q] = its x/y neighbours
    TX u[ZB + 2], nb[ZB][4];
    double s[ZB];
    double2 fv[ZB];
    const TX zero = {};
#pragma unroll
    for (int q = 0; q < ZB + 2; q++) {
        const int k = k0 - 1 + q;
        u[q] = k >= 0 && k < a.nz ? x[(q - 1) * plane] : zero;
    }
#pragma unroll
    for (int q = 0; q < ZB; q++) {
        const bool in = k0 + q < a.nz;
        const TX *xq = x + q * plane;
        nb[q][0] = in && hxm ? xq[-1] : zero;
        nb[q][1] = in && hxp ? xq[1] : zero;
        nb[q][2] = in && hym ? xq[-a.nx] : zero;
        nb[q][3] = in && hyp ? xq[a.nx] : zero;
        s[q] = in ? s2[q * plane] : 0.0;
        fv[q] = in && fin ? fin[q * plane] : make_double2(0, 0);
    }
    const double xs = a.xscale * (a.sc.p ? a.sc.p[r * a.sc.stride] : 1.0);

    // ---- per-axis couplings at this (i, j); for ADJ the ones that multiply the
    // neighbours are conj(cp[i-1]) (from i-1) and conj(cm[i+1]) (from i+1)
    double2 c_xm, c_xp, c_ym, c_yp, diag_xy;
    {
        const double2 cmx = a.cmx[i], cpx = a.cpx[i], cmy = a.cmy[j], cpy = a.cpy[j];
        diag_xy = make_double2(-(cmx.x + cpx.x + cmy.x + cpy.x), -(cmx.y + cpx.y + cmy.y + cpy.y));
        if (!ADJ) {
            c_xm = cmx;
            c_xp = cpx;
            c_ym = cmy;
            c_yp = cpy;
        } else {
            diag_xy.y = -diag_xy.y;
            c_xm = hxm ? a.cpx[i - 1] : make_double2(0, 0);
            c_xp = hxp ? a.cmx[i + 1] : make_double2(0, 0);
            c_ym = hym ? a.cpy[j - 1] : make_double2(0, 0);
            c_yp = hyp ? a.cmy[j + 1] : make_double2(0, 0);
            c_xm.y = -c_xm.y;
            c_xp.y = -c_xp.y;
            c_ym.y = -c_ym.y;
            c_yp.y = -c_yp.y;
        }
    }
    auto W = [](TX v) { return cvt<double2, TX>(v); };
#pragma unroll
    for (int q = 0; q < ZB; q++) {
        const int k = k0 + q;
        if (k >= a.nz) break;
        double2 czm, czp;
        const double2 cmz = a.cmz[k], cpz = a.cpz[k];
        double2 diag = make_double2(diag_xy.x - (cmz.x + cpz.x), diag_xy.y + (ADJ ? 1.0 : -1.0) * (cmz.y + cpz.y));
        if (!ADJ) {
            czm = cmz;
            czp = cpz;
        } else {
            czm = k > 0 ? a.cpz[k - 1] : make_double2(0, 0);
            czp = k + 1 < a.nz ? a.cmz[k + 1] : make_double2(0, 0);
            czm.y = -czm.y;
            czp.y = -czp.y;
        }
        // omega^2 s2 (1 + i beta), conjugated for the adjoint
        const double sw = a.w2 * s[q];
        diag.x += sw;
        diag.y += (ADJ ? -1.0 : 1.0) * sw * a.beta_phys;
        double2 acc = cmul(diag, W(u[q + 1]));
        if (hxm) acc = cfma(c_xm, W(nb[q][0]), acc);
        if (hxp) acc = cfma(c_xp, W(nb[q][1]), acc);
        if (hym) acc = cfma(c_ym, W(nb[q][2]), acc);
        if (hyp) acc = cfma(c_yp, W(nb[q][3]), acc);
        acc = cfma(czm, W(u[q]), acc);
        acc = cfma(czp, W(u[q + 2]), acc);
        acc.x *= xs;
        acc.y *= xs;
        if (fin) acc = make_double2(fv[q].x - acc.x, fv[q].y - acc.y);
        yout[q * plane] = acc;
    }
}

constexpr int kSbHX = kStX + 2, kSbHY = kStY + 2;

template <bool ADJ, typename TX, int ZB>
__global__ void __launch_bounds__(kStX *kStY, ZB <= 8 ? 4 : 2) stencil_block_kernel(StencilArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TX(*tile)[kSbHY][kSbHX] = reinterpret_cast<TX(*)[kSbHY][kSbHX]>(smem_raw);   // [ZB + 2]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = blockIdx.x * kStX, j0 = blockIdx.y * kStY;
    const int i = i0 + tx, j = j0 + ty;
    const int nzc = (a.nz + ZB - 1) / ZB;
    const int r = a.src_fast ? (int)(blockIdx.z % a.R) : (int)(blockIdx.z / nzc);
    const int zc = a.src_fast ? (int)(blockIdx.z / a.R) : (int)(blockIdx.z - r * nzc);
    const int k0 = zc * ZB;
    const long plane = (long)a.nx * a.ny;
    const TX *x = reinterpret_cast<const TX *>(a.x.p) + r * a.x.stride;
    // rows of the block with its halo: (plane, y) pairs, a warp per row
    for (int row = ty; row < (ZB + 2) * kSbHY; row += kStY) {
        const int hz = row / kSbHY, hy = row - hz * kSbHY;
        const int gk = k0 - 1 + hz, gj = j0 - 1 + hy;
        const bool line = gk >= 0 && gk < a.nz && gj >= 0 && gj < a.ny;
        const TX *src = x + (long)gk * plane + (long)gj * a.nx;
        const int gi = i0 - 1 + tx;
        const bool in = line && gi >= 0 && gi < a.nx;
        cp_async_el<sizeof(TX)>(&tile[hz][hy][tx], in ? src + gi : x, in);
        if (tx < kSbHX - kStX) {
            const bool in2 = line && gi + kStX < a.nx;
            cp_async_el<sizeof(TX)>(&tile[hz][hy][tx + kStX], in2 ? src + gi + kStX : x, in2);
        }
    }
    cp_async_commit();
    __shared__ double2 cz[ZB][3];   // couplings to k - 1 and k + 1, minus their diagonal part
    if (threadIdx.y == 0 && tx < ZB && k0 + tx < a.nz) {
        const int k = k0 + tx;
        const double2 cmz = a.cmz[k], cpz = a.cpz[k];
        double2 lo = cmz, hi = cpz;
        if (ADJ) {
            lo = k > 0 ? a.cpz[k - 1] : make_double2(0, 0);
            hi = k + 1 < a.nz ? a.cmz[k + 1] : make_double2(0, 0);
            lo.y = -lo.y;
            hi.y = -hi.y;
        }
        cz[tx][0] = lo;
        cz[tx][1] = hi;
        cz[tx][2] = make_double2(cmz.x + cpz.x, (ADJ ? -1.0 : 1.0) * (cmz.y + cpz.y));
    }
    const bool own = i < a.nx && j < a.ny;
    const long idx0 = (long)k0 * plane + (own ? (long)j * a.nx + i : 0);
    const double2 *fin = a.f.p ? a.f.p + r * a.f.stride + idx0 : nullptr;
    double2 *yout = a.y.p + r * a.y.stride + idx0;
    double s[ZB];
#pragma unroll
    for (int q = 0; q < ZB; q++) s[q] = own && k0 + q < a.nz ? a.s2[idx0 + q * plane] : 0.0;
    const double xs = a.xscale * (a.sc.p ? a.sc.p[r * a.sc.stride] : 1.0);
    double2 c_xm = make_double2(0, 0), c_xp = c_xm, c_ym = c_xm, c_yp = c_xm, diag_xy = c_xm;
    if (own) {   // as in stencil_kernel; off the grid the tile is zero
        const double2 cmx = a.cmx[i], cpx = a.cpx[i], cmy = a.cmy[j], cpy = a.cpy[j];
        diag_xy = make_double2(-(cmx.x + cpx.x + cmy.x + cpy.x), -(cmx.y + cpx.y + cmy.y + cpy.y));
        if (!ADJ) {
            c_xm = cmx;
            c_xp = cpx;
            c_ym = cmy;
            c_yp = cpy;
        } else {
            diag_xy.y = -diag_xy.y;
            c_xm = i > 0 ? a.cpx[i - 1] : make_double2(0, 0);
            c_xp = i + 1 < a.nx ? a.cmx[i + 1] : make_double2(0, 0);
            c_ym = j > 0 ? a.cpy[j - 1] : make_double2(0, 0);
            c_yp = j + 1 < a.ny ? a.cmy[j + 1] : make_double2(0, 0);
            c_xm.y = -c_xm.y;
            c_xp.y = -c_xp.y;
            c_ym.y = -c_ym.y;
            c_yp.y = -c_yp.y;
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    if (!own) return;
    auto T = [&](int b, int hy, int hx) { return cvt<double2, TX>(tile[b][hy][hx]); };
    double2 um = T(0, ty + 1, tx + 1), uc = T(1, ty + 1, tx + 1);
#pragma unroll
    for (int q = 0; q < ZB; q++) {
        const int k = k0 + q;
        if (k >= a.nz) break;
        const double2 up = T(q + 2, ty + 1, tx + 1);
        const double2 czm = cz[q][0], czp = cz[q][1];
        double2 diag = csub(diag_xy, cz[q][2]);
        const double sw = a.w2 * s[q];
        diag.x += sw;
        diag.y += (ADJ ? -1.0 : 1.0) * sw * a.beta_phys;
        double2 acc = cmul(diag, uc);
        acc = cfma(c_xm, T(q + 1, ty + 1, tx), acc);
        acc = cfma(c_xp, T(q + 1, ty + 1, tx + 2), acc);
        acc = cfma(c_ym, T(q + 1, ty, tx + 1), acc);
        acc = cfma(c_yp, T(q + 1, ty + 2, tx + 1), acc);
        acc = cfma(czm, um, acc);
        acc = cfma(czp, up, acc);
        acc.x *= xs;
        acc.y *= xs;
        if (fin) {
            const double2 fv = fin[q * plane];
            acc = make_double2(fv.x - acc.x, fv.y - acc.y);
        }
        yout[q * plane] = acc;
        um = uc;
        uc = up;
    }
}

template <typename TX, int ZB, bool BLOCK> static int stencil_go(const StencilArgs &a, bool adjoint, cudaStream_t s) {
    dim3 block(kStX, kStY);
    dim3 grid((a.nx + kStX - 1) / kStX, (a.ny + kStY - 1) / kStY, ((a.nz + ZB - 1) / ZB) * a.R);
    if constexpr (BLOCK) {
        const size_t smem = (size_t)(ZB + 2) * kSbHY * kSbHX * sizeof(TX);
        void (*kern)(StencilArgs) = adjoint ? stencil_block_kernel<true, TX, ZB> : stencil_block_kernel<false, TX, ZB>;
        if (smem > 48 * 1024 && !smem_limit_max(kern, smem)) return HELM3D_ERR_CUDA;
        kern<<<grid, block, smem, s>>>(a);
    } else {
        if (adjoint) stencil_kernel<true, TX, ZB><<<grid, block, 0, s>>>(a);
        else stencil_kernel<false, TX, ZB><<<grid, block, 0, s>>>(a);
    }
    return cudaGetLastError() == cudaSuccess ? HELM3D_OK : HELM3D_ERR_CUDA;
}

template <typename TX> static int stencil_zb(const StencilArgs &a, bool adjoint, cudaStream_t s) {
    switch (a.zblock) {
        case 1: return stencil_go<TX, 1, false>(a, adjoint, s);
        case 2: return stencil_go<TX, 2, false>(a, adjoint, s);
        case 4: return stencil_go<TX, 4, true>(a, adjoint, s);
        case 6: return stencil_go<TX, 6, true>(a, adjoint, s);
        case 8: return stencil_go<TX, 8, true>(a, adjoint, s);
        case 12: return stencil_go<TX, 12, true>(a, adjoint, s);
    }
    return HELM3D_ERR_ARG;
}

// The z points per thread of an untuned launch: blocks of 8 planes where they
// occupy every SM four times (200^3: 117 -> 83 us with the old marching kernel's
// best at 106; blocks of 4 planes 91, the register kernel 132), fewer planes on
// smaller grids (96^3, 6 planes: 17.5 -> 15.0), the register kernel where even 4
// leave SMs idle (20^3: 22 -> 8.5 us, 4 planes 10.8; all with some 5 us of events).
int stencil_default(int nx, int ny, int nz, int R) {
    const long cols = (long)((nx + kStX - 1) / kStX) * ((ny + kStY - 1) / kStY) * R, sms = device_info().sm_count;
    auto blocks = [&](int zb) { return cols * ((nz + zb - 1) / zb); };
    if (blocks(8) >= 4 * sms) return 8;
    if (2 * blocks(6) >= 5 * sms) return 6;
    return blocks(4) >= sms ? 4 : 1;
}

int launch_stencil(const StencilArgs &a, bool adjoint, cudaStream_t s) {
    if (a.y.c64 || a.f.c64) return HELM3D_ERR_ARG;
    return a.x.c64 ? stencil_zb<float2>(a, adjoint, s) : stencil_zb<double2>(a, adjoint, s);
}

}  // namespace h3d
