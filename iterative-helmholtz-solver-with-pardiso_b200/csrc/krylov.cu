// krylov.cu -- complex128 vector kernels of the outer Krylov loop: the
// Gram-Schmidt dot products and updates (the reference's zdotc/zaxpy loop,
// Source/FGMRES.cpp:508-517), norms (dznrm2, :519; the physical-domain norm
// after reducePML3D, :590-592), the solution update x = x0 + Z y (zgemv,
// :575) and small helpers.  Every kernel takes a batch of R right-hand sides
// (blockIdx.y = r, per-r pointer strides).  Reductions are two-level and
// deterministic: a partial per block, then one pass over them by the block that
// finishes last, which also does the step's bookkeeping (arnoldi.cuh).
#include <cuda_runtime.h>

#include "arnoldi.cuh"
#include "cplx.cuh"
#include "helm3d_internal.h"

namespace h3d {

constexpr int kRedThreads = 256;
constexpr int kRedWarps = kRedThreads / 32;

// Whether this block is the last of n to get here on `ticket` (zero between
// launches): its threads then see what every other block wrote before.
__device__ __forceinline__ bool last_to_finish(int *ticket, int n) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(ticket, 1) == n - 1;
        if (last) *ticket = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// sum of the nb partials at part, by a warp (fixed order: deterministic), 8
// loads in flight per lane
__device__ __forceinline__ double2 sum_partials(const double2 *part, int nb) {
    double2 s = make_double2(0, 0);
    for (int b0 = threadIdx.x & 31; b0 < nb; b0 += 256) {
        double2 q[8];
#pragma unroll
        for (int u = 0; u < 8; u++) q[u] = b0 + 32 * u < nb ? __ldcg(part + b0 + 32 * u) : make_double2(0, 0);
#pragma unroll
        for (int u = 0; u < 8; u++) s = cadd(s, q[u]);
    }
    return warp_sum(s);
}

// the sum over the block of one complex value per thread; valid in thread 0
__device__ __forceinline__ double2 block_sum(double2 v) {
    __shared__ double2 sh[kRedWarps];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kRedWarps; w++) v = cadd(v, sh[w]);
    return v;
}

// What follows a pass, in the block of a right-hand side that finishes last
// (arnoldi.cuh), and, where it concerns the batch, in the last of those.
enum KryEnd {
    KE_NONE = 0,      // the sums only
    KE_LAGGED = 1,    // dots of DCGS2's step j: column j - 1, the update coefficients
    KE_TAIL = 2,      // dots of the cycle's last vector: the open column, then y = R^{-1} g
    KE_BACKSUB = 3,   // no dots: y = R^{-1} g
    KE_POST = 4,      // DCGS2's update: scale of V_{j+1}, whether step j + 1 runs
    KE_REORTH = 5,    // classical Gram-Schmidt's first update: whether a second pass is needed
    KE_GIVENS = 6     // its second (possibly skipped) update: column j, whether step j + 1 runs
};

struct DotsK {
    const double2 *V;
    long ldv, sV;
    const double *vs;
    long sVs;
    int nv, norm;             // basis vectors; with norm also ||w||^2
    const double2 *w;
    long sW, N;
    double2 *partials;        // of right-hand side r at r * sPart, slot s at s * blocks
    long sPart;
    int *tickets;             // [R] per right-hand side, then one for the batch
    double2 *out;
    long sOut;
    const int *pred;          // when given and *pred == 0: no pass
    int end, j;
    ArnState arn;
};

constexpr int kDotVecs = 64;   // vectors whose sums a block keeps in shared memory at a time

// sums over the warp of NV (2 or 4) values per lane, by halving: the lanes with
// (lane & (64 / NV - 1 >> 1)) == 0 hold value number dot_slot<NV>(lane)
template <int NV> __device__ __forceinline__ int dot_slot(int lane) { return NV == 4 ? lane >> 3 : lane >> 4; }
template <int NV> __device__ __forceinline__ double reduce_values(const double (&v)[NV], int lane) {
    double c;
    if constexpr (NV == 4) {
        const bool hi = lane & 16, hi2 = lane & 8;
        double a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
        a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
        b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
        c = hi2 ? b : a;
        c += __shfl_xor_sync(0xffffffffu, hi2 ? a : b, 8);
    } else {
        const bool hi = lane & 16;
        c = hi ? v[1] : v[0];
        c += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[1], 16);
        c += __shfl_xor_sync(0xffffffffu, c, 8);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    return c;
}

// The dots of `items` vectors (V_0 .. V_{nv-1}, then w itself for its norm)
// with w, and with TWO also with V_j = V_{nv-1} (DCGS2's lagged second
// projection).  A warp takes tiles of 32 UL values of l, keeps w and V_j of the
// tile in registers and goes through the vectors, 8 / UL at a time (8 loads in
// flight per lane); a vector's sums over the tile are reduced by halving (6
// shuffles for 4 values) and added to the warp's in shared memory.  So w and
// V_j are read once whatever the number of vectors, every warp has the same
// work, and no thread keeps more than a batch of sums (one thread per l for
// all vectors kept 18: 126 registers, two CTAs per SM, 180 shuffles a block).
// UL = 4 where the tiles outnumber the warps, less on small grids.
template <bool TWO, int UL>
__global__ void __launch_bounds__(kRedThreads) dots_kernel(DotsK a) {
    constexpr int VB = 8 / UL, NV = TWO ? 4 : 2;
    __shared__ double sacc[kRedWarps][kDotVecs][NV];
    extern __shared__ __align__(16) double2 sm[];
    const int r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int nv = a.nv;
    const double2 *V = a.V + r * a.sV, *w = a.w + r * a.sW;
    bool pass = !(a.pred && *a.pred == 0);
    if (a.end == KE_LAGGED || a.end == KE_TAIL) pass = pass && !a.arn.frozen[r];
    if (a.end == KE_TAIL) {   // the number of steps a graph ran is known on the device only
        nv = a.arn.flags[4] + 1;
        w = V + (long)nv * a.ldv;
    }
    if (!pass && (a.end != KE_TAIL || blockIdx.x > 0)) return;
    const int items = nv + a.norm, nb = gridDim.x;
    double2 *part = a.partials + r * a.sPart;
    if (pass) {
        const double2 *x2 = V + (long)(nv - 1) * a.ldv;
        for (int c0 = 0; c0 < items; c0 += kDotVecs) {
            const int nc = min(items - c0, kDotVecs);
            double *mine = &sacc[warp][0][0];
            for (int q = lane; q < nc * NV; q += 32) mine[q] = 0.0;
            __syncwarp();
            const long step = (long)nb * kRedWarps * (32 * UL);
            for (long t0 = ((long)blockIdx.x * kRedWarps + warp) * (32 * UL); t0 < a.N; t0 += step) {
                const long l = t0 + lane;
                const bool whole = t0 + 32 * UL <= a.N;
                double2 wv[UL], xv[UL];
#pragma unroll
                for (int u = 0; u < UL; u++) {
                    const bool in = whole || l + 32 * u < a.N;
                    wv[u] = in ? w[l + 32 * u] : make_double2(0, 0);
                    xv[u] = TWO && in ? x2[l + 32 * u] : make_double2(0, 0);
                }
                for (int i0 = 0; i0 < nc; i0 += VB) {
                    double2 v[VB][UL];
#pragma unroll
                    for (int q = 0; q < VB; q++) {
                        const int i = c0 + i0 + q;
                        const double2 *p = i < nv ? V + (long)i * a.ldv : w;
#pragma unroll
                        for (int u = 0; u < UL; u++)
                            v[q][u] = i0 + q < nc && (whole || l + 32 * u < a.N) ? p[l + 32 * u] : make_double2(0, 0);
                    }
#pragma unroll
                    for (int q = 0; q < VB; q++) {
                        double s[NV];
#pragma unroll
                        for (int e = 0; e < NV; e++) s[e] = 0.0;
#pragma unroll
                        for (int u = 0; u < UL; u++) {   // conj(v) w, conj(v) x2
                            s[0] = fma(v[q][u].y, wv[u].y, fma(v[q][u].x, wv[u].x, s[0]));
                            s[1] = fma(-v[q][u].y, wv[u].x, fma(v[q][u].x, wv[u].y, s[1]));
                            if constexpr (TWO) {
                                s[2] = fma(v[q][u].y, xv[u].y, fma(v[q][u].x, xv[u].x, s[2]));
                                s[3] = fma(-v[q][u].y, xv[u].x, fma(v[q][u].x, xv[u].y, s[3]));
                            }
                        }
                        const double c = reduce_values<NV>(s, lane);
                        if ((lane & (32 / NV - 1)) == 0 && i0 + q < nc) mine[(i0 + q) * NV + dot_slot<NV>(lane)] += c;
                    }
                }
            }
            __syncthreads();
            // the block's sums: slot i <V_i, w>, with TWO slot nv + i <V_i, V_j>
            for (int q = threadIdx.x; q < nc * NV; q += kRedThreads) {
                double s = 0.0;
#pragma unroll
                for (int u = 0; u < kRedWarps; u++) s += (&sacc[u][0][0])[q];
                const int i = c0 + q / NV, e = q % NV;
                double2 *p = part + (long)(e < 2 ? i : nv + i) * nb + blockIdx.x;
                if (e & 1) p->y = s;
                else p->x = s;
            }
            if (c0 + kDotVecs < items) __syncthreads();
        }
        if (!last_to_finish(a.tickets + r, nb)) return;
        // slots 0 .. nv-1: vs_i <V_i, w>; then ||w||^2, or with TWO
        // vs_i <V_i, V_j> (i < j) and <V_j, V_j>
        const double *vs = a.vs ? a.vs + r * a.sVs : nullptr;
        const int slots = TWO ? 2 * nv : items;
        for (int s = warp; s < slots; s += kRedWarps) {
            double2 t = sum_partials(part + (long)s * nb, nb);
            const int i = s < nv ? s : TWO && s < 2 * nv - 1 ? s - nv : -1;
            if (vs && i >= 0) t = cscale(t, vs[i]);
            if (lane == 0) {
                if (a.out) a.out[r * a.sOut + s] = t;
                if (a.end != KE_NONE) sm[s] = t;
            }
        }
        if (a.end == KE_NONE) return;
        __syncthreads();
        if (a.end == KE_LAGGED) {
            if (warp == 0) lagged_step(a.arn, r, a.j, sm, sm + slots);
            return;
        }
    }
    // KE_TAIL: the open column (of a right-hand side still active), then y
    if (pass && warp == 0) lagged_final(a.arn, r, nv, sm, sm + items);
    __syncthreads();
    backsub_block(a.arn, r, sm, sm + a.arn.m);
    if (last_to_finish(a.tickets + gridDim.y, gridDim.y) && warp == 0) {
        // the longest column count of the batch
        int k = 0;
        for (int p = lane; p < a.arn.B; p += 32) k = max(k, __ldcg(a.arn.k + p));
        for (int off = 16; off > 0; off >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, off));
        if (lane == 0) a.arn.flags[2] = k;
    }
}

// y = R^{-1} g of every right-hand side (a block each), without dots
__global__ void __launch_bounds__(kRedThreads) backsub_kernel(ArnState a, int *ticket) {
    extern __shared__ __align__(16) double2 sm[];
    const int lane = threadIdx.x & 31;
    backsub_block(a, blockIdx.x, sm, sm + a.m);
    if (last_to_finish(ticket, gridDim.x) && threadIdx.x < 32) {
        int k = 0;
        for (int p = lane; p < a.B; p += 32) k = max(k, __ldcg(a.k + p));
        for (int off = 16; off > 0; off >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, off));
        if (lane == 0) a.flags[2] = k;
    }
}

struct UpdateK {
    double2 *V;
    long ldv, sV;
    const double *vs;         // classical Gram-Schmidt: basis scales, or null
    long sVs;
    int nv;                   // basis vectors; DCGS2: j
    const double2 *coef;
    long sCoef;
    int M2;
    double2 *w;
    long sW, N;
    int post;                 // ||w||^2 into out[r].x
    double2 *partials;
    long sPart;
    int *tickets;
    double2 *out;
    long sOut;
    const int *pred;
    int end, j, has_next;
    cudaGraphConditionalHandle next;
    ArnState arn;
};

// What follows an update pass: the norm from the blocks' partials (its own in
// `nrm`; with !pass none was taken), then the end of the step.  Every block
// gets here with `pass`; without it only block 0 of each right-hand side.
template <bool GIVENS> __device__ __forceinline__ void update_end(const UpdateK &a, int r, bool pass, double2 nrm, double2 *scr) {
    if (pass) {
        if (threadIdx.x == 0) a.partials[r * a.sPart + blockIdx.x] = nrm;
        if (!last_to_finish(a.tickets + r, gridDim.x)) return;
        if (threadIdx.x < 32) {
            nrm = sum_partials(a.partials + r * a.sPart, gridDim.x);
            if (threadIdx.x == 0) a.out[r * a.sOut] = nrm;
        }
    }
    if (a.end == KE_NONE) return;
    if (threadIdx.x < 32) {
        __syncwarp();
        if (!GIVENS && threadIdx.x == 0) post_step(a.arn, r, a.j, pass ? nrm.x : 0.0);
        if (GIVENS && a.end == KE_GIVENS) givens_step(a.arn, r, a.j, scr);
    }
    if (!last_to_finish(a.tickets + gridDim.y, gridDim.y) || threadIdx.x >= 32) return;
    // the batch: is some right-hand side still active / in need of a second pass
    int any = 0;
    for (int p = threadIdx.x; p < a.arn.B; p += 32) {
        if (__ldcg(a.arn.frozen + p)) continue;
        const double2 *h = a.arn.h + (long)p * a.arn.SH;
        any |= a.end != KE_REORTH || __ldcg(&h[2 * a.arn.M2].x) < H3D_REORTH_ETA2 * __ldcg(&h[a.j + 1].x);
    }
    any = __any_sync(0xffffffffu, any);
    if (threadIdx.x > 0) return;
    if (a.end == KE_REORTH) {
        a.arn.flags[0] = any;
        if (any) a.arn.flags[1] += 1;
    } else {
        a.arn.flags[4] = a.j;
        a.arn.flags[5] = any;
        if (a.has_next) cudaGraphSetConditional(a.next, any ? 1u : 0u);
    }
}

// w -= sum_i coef[i] vs[i] V_i, with post ||w_new||^2
__global__ void __launch_bounds__(kRedThreads) update_kernel(UpdateK a) {
    extern __shared__ __align__(16) double2 sc[];  // nv coefficients (coef * vs), then the scratch of the step's end
    const int r = blockIdx.y;
    const bool pass = !(a.pred && *a.pred == 0);
    if (!pass && (blockIdx.x > 0 || a.end == KE_NONE)) return;
    double2 nrm = make_double2(0, 0);
    if (pass) {
        const double2 *V = a.V + r * a.sV, *coef = a.coef + r * a.sCoef;
        const double *vs = a.vs ? a.vs + r * a.sVs : nullptr;
        double2 *w = a.w + r * a.sW;
        for (int i = threadIdx.x; i < a.nv; i += blockDim.x) sc[i] = cscale(coef[i], vs ? vs[i] : 1.0);
        __syncthreads();
        const long stride = (long)gridDim.x * blockDim.x;
        for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < a.N; l += stride) {
            double2 acc = w[l];
            int i = 0;
            // 8 basis loads in flight ahead of their FMAs (58^3: 23 -> 14 us a pass)
            for (; i + 8 <= a.nv; i += 8) {
                double2 v[8];
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = V[(long)(i + q) * a.ldv + l];
#pragma unroll
                for (int q = 0; q < 8; q++) acc = cfms(sc[i + q], v[q], acc);
            }
            if (i < a.nv) {
                double2 v[7];
#pragma unroll
                for (int q = 0; q < 7; q++) v[q] = i + q < a.nv ? V[(long)(i + q) * a.ldv + l] : make_double2(0, 0);
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (i + q < a.nv) acc = cfms(sc[i + q], v[q], acc);
            }
            w[l] = acc;
            nrm.x += acc.x * acc.x + acc.y * acc.y;
        }
        if (!a.post) return;
        nrm = block_sum(nrm);
    }
    update_end<true>(a, r, pass, nrm, sc);
}

// The DCGS2 update pass: with alpha = coef[0 .. j-1], delta = coef[M2 .. M2+j]
//   V_j <- V_j - sum_{i<j} alpha_i V_i                 (j > 0)
//   w   <- w - sum_{i<j} delta_i V_i - delta_j V_j(old)
// and ||w||^2; a frozen right-hand side: nothing read or written but its state.
// U > 1: the basis loads of U consecutive i issued together ahead of their
// FMAs (more bytes in flight per thread; the FMA order, and so the result,
// is the same as U = 1).
template <int U>
__global__ void __launch_bounds__(kRedThreads) update2_kernel(UpdateK a) {
    extern __shared__ __align__(16) double2 sc[];  // alpha[j], delta[j + 1]
    const int r = blockIdx.y, j = a.nv;
    const bool pass = !(a.end == KE_POST && a.arn.frozen[r]);
    if (!pass && blockIdx.x > 0) return;
    double2 nrm = make_double2(0, 0);
    if (pass) {
        double2 *V = a.V + r * a.sV, *w = a.w + r * a.sW;
        const double2 *coef = a.coef + r * a.sCoef;
        double2 *alpha = sc, *delta = sc + j;
        for (int i = threadIdx.x; i < j; i += blockDim.x) alpha[i] = coef[i];
        for (int i = threadIdx.x; i <= j; i += blockDim.x) delta[i] = coef[a.M2 + i];
        __syncthreads();
        double2 *__restrict__ vj = V + (long)j * a.ldv;
        const long stride = (long)gridDim.x * blockDim.x;
        for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < a.N; l += stride) {
            double2 x = vj[l];
            double2 acc = cfms(delta[j], x, w[l]);
            int i = 0;
            if (U > 1) {
                for (; i + U <= j; i += U) {
                    double2 v[U];
#pragma unroll
                    for (int q = 0; q < U; q++) v[q] = V[(long)(i + q) * a.ldv + l];
#pragma unroll
                    for (int q = 0; q < U; q++) {
                        x = cfms(alpha[i + q], v[q], x);
                        acc = cfms(delta[i + q], v[q], acc);
                    }
                }
            }
            if (U > 1) {
                if (i < j) {   // the rest, likewise
                    double2 v[U - 1 > 0 ? U - 1 : 1];
#pragma unroll
                    for (int q = 0; q < U - 1; q++) v[q] = i + q < j ? V[(long)(i + q) * a.ldv + l] : make_double2(0, 0);
#pragma unroll
                    for (int q = 0; q < U - 1; q++)
                        if (i + q < j) {
                            x = cfms(alpha[i + q], v[q], x);
                            acc = cfms(delta[i + q], v[q], acc);
                        }
                }
            } else {
                for (; i < j; i++) {
                    const double2 v = V[(long)i * a.ldv + l];
                    x = cfms(alpha[i], v, x);
                    acc = cfms(delta[i], v, acc);
                }
            }
            if (j > 0) vj[l] = x;
            w[l] = acc;
            nrm.x += acc.x * acc.x + acc.y * acc.y;
        }
        nrm = block_sum(nrm);
    }
    update_end<false>(a, r, pass, nrm, sc);
}

__global__ void cycle_init_kernel(ArnState a, CycleInit ci) {
    const int p = threadIdx.x;
    if (p < kArnFlags) a.flags[p] = 0;
    if (p >= a.B) return;
    a.nf[p] = ci.nf[p];
    a.tol[p] = ci.tol;
    a.it[p] = ci.it[p];
    a.max_iter[p] = ci.max_iter;
    a.frozen[p] = a.k[p] = 0;
    a.g[(long)p * (a.m + 1)] = make_double2(ci.beta[p], 0.0);
    a.vs[(long)p * a.M2] = 1.0 / ci.beta[p];
}

// x += sum_i y[i] zs[i] Z_i  (i < *nzv_dev when given, else nzv); Z complex128 or complex64
template <typename TZ>
__global__ void __launch_bounds__(kRedThreads) combine_kernel(const TZ *__restrict__ Z, long ldz, long sZ,
                                                              const double *__restrict__ zs, long sZs, int nzv,
                                                              const double2 *__restrict__ y, long sY,
                                                              double2 *__restrict__ x, long sX, long N,
                                                              const int *nzv_dev) {
    extern __shared__ double2 sc[];
    if (nzv_dev) nzv = min(nzv, *nzv_dev);
    const int r = blockIdx.y;
    Z += r * sZ;
    y += r * sY;
    x += r * sX;
    if (zs) zs += r * sZs;
    for (int i = threadIdx.x; i < nzv; i += blockDim.x) sc[i] = cscale(y[i], zs ? zs[i] : 1.0);
    __syncthreads();
    const long stride = (long)gridDim.x * blockDim.x;
    for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += stride) {
        double2 acc = x[l];
        for (int i = 0; i < nzv; i += 8) {   // 8 loads in flight ahead of their FMAs
            TZ z[8];
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (i + q < nzv) z[q] = Z[(long)(i + q) * ldz + l];
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (i + q < nzv) acc = cfma(sc[i + q], cvt<double2, TZ>(z[q]), acc);
        }
        x[l] = acc;
    }
}

// out[r * sOut].x = ||x_r||^2 over the whole grid and, with phys,
// out[r * sOut + 1].x over the box [x0, x1) x [y0, y1) x [z0, z1), in one pass:
// a warp per grid line
struct NormK {
    const double2 *x;
    long sX;
    int nx, ny, nz, box[6], phys;
    double2 *partials;
    long sPart;
    int *tickets;
    double2 *out;
    long sOut;
};
__global__ void __launch_bounds__(kRedThreads) norm2_kernel(NormK a) {
    const int r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double2 *x = a.x + r * a.sX;
    double2 acc = make_double2(0, 0);   // whole grid, box
    const int lines = a.ny * a.nz;
    for (int q = blockIdx.x * kRedWarps + warp; q < lines; q += gridDim.x * kRedWarps) {
        const int k = q / a.ny, j = q - k * a.ny;
        const bool in = j >= a.box[2] && j < a.box[3] && k >= a.box[4] && k < a.box[5];
        const double2 *xl = x + (long)q * a.nx;
        for (int i = lane; i < a.nx; i += 32) {
            const double2 v = xl[i];
            const double s = v.x * v.x + v.y * v.y;
            acc.x += s;
            if (in && i >= a.box[0] && i < a.box[1]) acc.y += s;
        }
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) a.partials[r * a.sPart + blockIdx.x] = acc;
    if (!last_to_finish(a.tickets + r, gridDim.x) || threadIdx.x >= 32) return;
    acc = sum_partials(a.partials + r * a.sPart, gridDim.x);
    if (lane == 0) {
        a.out[r * a.sOut] = make_double2(acc.x, 0);
        if (a.phys) a.out[r * a.sOut + 1] = make_double2(acc.y, 0);
    }
}

__global__ void axpby_kernel(double2 a, const double2 *__restrict__ x, long sX, double2 b, double2 *__restrict__ y,
                             long sY, long N) {
    const int r = blockIdx.y;
    x += r * sX;
    y += r * sY;
    const long stride = (long)gridDim.x * blockDim.x;
    for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += stride) {
        const double2 yv = y[l], xv = x[l];
        y[l] = cadd(cmul(a, xv), cmul(b, yv));
    }
}

__global__ void sub_dl_kernel(const double2 *__restrict__ x, const double2 *__restrict__ dl,
                              const double2 *__restrict__ t, double2 *__restrict__ y, long N) {
    const long stride = (long)gridDim.x * blockDim.x;
    for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += stride) y[l] = csub(x[l], cmul(dl[l], t[l]));
}

// vs[r][j] = 1 / sqrt(nrm[r].x)
__global__ void set_scale_kernel(const double2 *nrm, long sNrm, double *vs, long sVs, int j, int R) {
    const int r = threadIdx.x;
    if (r < R) {
        const double s = sqrt(nrm[r * sNrm].x);
        vs[r * sVs + j] = s > 0 ? 1.0 / s : 0.0;
    }
}

template <typename R>
__global__ void base2d_kernel(const double *__restrict__ s2, int nz, long plane, int zlo, int zhi, double w2,
                              double beta, cplx<R> *__restrict__ out, int *status) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= plane) return;
    double s = 0.0;
    bool bad = false;
    for (int k = 0; k < nz; k++) {
        const double v = s2[(long)k * plane + q];
        bad |= !isfinite(v);
        if (k >= zlo && k < zhi) s += v;
    }
    s *= w2 / (double)(zhi - zlo);
    out[q] = cvt<cplx<R>, double2>(make_double2(s, s * beta));
    if (bad) atomicOr(status, 16);
}

static inline bool ok() { return cudaGetLastError() == cudaSuccess; }

// Dynamic shared memory above this is opted in to: with the kernel's own (up to
// 16 KB of sums in dots_kernel, 144 bytes in the others) it may pass the 48 KB
// that a launch gets without.
constexpr size_t kSmemOptIn = 24 * 1024;

static int grid_for(long N, int R = 1) {
    const long b = (N + kRedThreads - 1) / kRedThreads;
    const long cap = (4L * device_info().sm_count + R - 1) / R;
    return (int)(b < cap ? (b < 1 ? 1 : b) : (cap < 1 ? 1 : cap));
}

// blocks of a pass: the tuned number, but no more than blocks of `per` values
static int pass_blocks(const Reduce &red, long N, int per) {
    const long b = (N + per - 1) / per;
    return (int)(b < red.nblocks ? (b < 1 ? 1 : b) : red.nblocks);
}

static int go_dots(const DotsK &a, int items, bool two, const Reduce &red, int R, size_t scratch, cudaStream_t s) {
    if (items * (two ? 2 : 1) > red.cap || R > red.rmax) return HELM3D_ERR_ARG;
    const size_t smem = sizeof(double2) * scratch;
    auto go = [&](void (*kern)(DotsK), int ul) -> int {
        if (smem > kSmemOptIn && !smem_limit_max(kern, smem)) return HELM3D_ERR_CUDA;
        kern<<<dim3(pass_blocks(red, a.N, 32 * ul * kRedWarps), R), kRedThreads, smem, s>>>(a);
        return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
    };
    // tiles per warp of the tuned grid: the largest tile that leaves every warp
    // four, so that the last round of tiles is a small part of the pass
    const long warps = (long)red.nblocks * kRedWarps;
    if (a.N >= warps * 128 * 4) return two ? go(dots_kernel<true, 4>, 4) : go(dots_kernel<false, 4>, 4);
    if (a.N >= warps * 64 * 4) return two ? go(dots_kernel<true, 2>, 2) : go(dots_kernel<false, 2>, 2);
    return two ? go(dots_kernel<true, 1>, 1) : go(dots_kernel<false, 1>, 1);
}

static DotsK dots_args(const VecBatch &V, long ldv, const ScaleBatch &vs, int nv, bool norm, const VecBatch &w, long N,
                       const Reduce &red, double2 *out, long sOut) {
    DotsK a = {};
    a.V = V.p;
    a.ldv = ldv;
    a.sV = V.stride;
    a.vs = vs.p;
    a.sVs = vs.stride;
    a.nv = nv;
    a.norm = norm ? 1 : 0;
    a.w = w.p;
    a.sW = w.stride;
    a.N = N;
    a.partials = red.partials;
    a.sPart = red.stride;
    a.tickets = red.tickets;
    a.out = out;
    a.sOut = sOut;
    return a;
}

int launch_dots(const VecBatch &V, long ldv, const ScaleBatch &vs, int nv, const VecBatch &w, long N, int R,
                const Reduce &red, double2 *out, long sOut, cudaStream_t s, bool wnorm, const int *pred) {
    DotsK a = dots_args(V, ldv, vs, nv, wnorm, w, N, red, out, sOut);
    a.pred = pred;
    return go_dots(a, nv + (wnorm ? 1 : 0), false, red, R, 0, s);
}

int launch_dots2(const VecBatch &V, long ldv, const ScaleBatch &vs, int j, const VecBatch &w, long N, int R,
                 const Reduce &red, double2 *out, long sOut, cudaStream_t s, const ArnState *arn) {
    DotsK a = dots_args(V, ldv, vs, j + 1, false, w, N, red, out, sOut);
    if (arn) {
        a.end = KE_LAGGED;
        a.j = j;
        a.arn = *arn;
    }
    return go_dots(a, j + 1, true, red, R, arn ? arn_scratch(j) : 0, s);
}

int launch_cycle_end(const VecBatch &V, long ldv, const ArnState &arn, bool tail, long N, int R, const Reduce &red,
                     cudaStream_t s) {
    const size_t scratch = arn_scratch(arn.m + 1) + kBacksubTri * kBacksubTri;
    if (!tail) {
        const size_t smem = sizeof(double2) * scratch;
        if (smem > kSmemOptIn && !smem_limit_max(backsub_kernel, smem)) return HELM3D_ERR_CUDA;
        backsub_kernel<<<R, kRedThreads, smem, s>>>(arn, red.tickets + red.rmax);
        return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
    }
    DotsK a = dots_args(V, ldv, ScaleBatch{arn.vs, arn.M2}, 0, true, V, N, red, nullptr, 0);
    a.pred = arn.flags + 5;   // none active: every column is closed
    a.end = KE_TAIL;
    a.arn = arn;
    return go_dots(a, arn.m + 1, false, red, R, scratch, s);
}

static UpdateK update_args(const VecBatch &V, long ldv, int nv, const double2 *coef, long sCoef, const VecBatch &w,
                           long N, const Reduce &red, double2 *out, long sOut) {
    UpdateK a = {};
    a.V = V.p;
    a.ldv = ldv;
    a.sV = V.stride;
    a.nv = nv;
    a.coef = coef;
    a.sCoef = sCoef;
    a.w = w.p;
    a.sW = w.stride;
    a.N = N;
    a.partials = red.partials;
    a.sPart = red.stride;
    a.tickets = red.tickets;
    a.out = out;
    a.sOut = sOut;
    return a;
}

int launch_update(const VecBatch &V, long ldv, const ScaleBatch &vs, int nv, const double2 *coef, long sCoef,
                  const VecBatch &w, long N, int R, int post, const Reduce &red, double2 *out, long sOut,
                  cudaStream_t s, const int *pred, const ArnState *arn, int j, bool has_next,
                  cudaGraphConditionalHandle next) {
    if (R > red.rmax) return HELM3D_ERR_ARG;
    UpdateK a = update_args(V, ldv, nv, coef, sCoef, w, N, red, out, sOut);
    a.vs = vs.p;
    a.sVs = vs.stride;
    a.post = post;
    a.pred = pred;
    a.j = j;
    a.has_next = has_next ? 1 : 0;
    a.next = next;
    if (arn) {
        a.end = pred ? KE_GIVENS : KE_REORTH;
        a.arn = *arn;
    }
    const int nb = post ? pass_blocks(red, N, kRedThreads) : grid_for(N, R);
    const size_t smem = sizeof(double2) * (arn ? arn_scratch(nv) : nv > 0 ? (size_t)nv : 1);
    if (smem > kSmemOptIn && !smem_limit_max(update_kernel, smem)) return HELM3D_ERR_CUDA;
    update_kernel<<<dim3(nb, R), kRedThreads, smem, s>>>(a);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_update2(const VecBatch &V, long ldv, int j, const double2 *coef, long sCoef, int M2, const VecBatch &w,
                   long N, int R, const Reduce &red, double2 *out, long sOut, cudaStream_t s, const ArnState *arn,
                   bool has_next, cudaGraphConditionalHandle next) {
    if (R > red.rmax) return HELM3D_ERR_ARG;
    UpdateK a = update_args(V, ldv, j, coef, sCoef, w, N, red, out, sOut);
    a.M2 = M2;
    a.j = j;
    a.has_next = has_next ? 1 : 0;
    a.next = next;
    if (arn) {
        a.end = KE_POST;
        a.arn = *arn;
    }
    const dim3 grid(pass_blocks(red, N, kRedThreads), R);
    const size_t smem = sizeof(double2) * (2 * j + 1);
    if (red.update == 1) update2_kernel<8><<<grid, kRedThreads, smem, s>>>(a);
    else update2_kernel<1><<<grid, kRedThreads, smem, s>>>(a);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_combine(const VecBatch &Z, long ldz, const ScaleBatch &zs, int nzv, const double2 *y, long sY,
                   const VecBatch &x, long N, int R, cudaStream_t s, const int *nzv_dev) {
    const dim3 grid(grid_for(N, R), R);
    const size_t sm = sizeof(double2) * (nzv > 0 ? nzv : 1);
    if (Z.c64)
        combine_kernel<float2><<<grid, kRedThreads, sm, s>>>(reinterpret_cast<const float2 *>(Z.p), ldz, Z.stride,
                                                             zs.p, zs.stride, nzv, y, sY, x.p, x.stride, N, nzv_dev);
    else
        combine_kernel<double2><<<grid, kRedThreads, sm, s>>>(Z.p, ldz, Z.stride, zs.p, zs.stride, nzv, y, sY, x.p,
                                                              x.stride, N, nzv_dev);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_cycle_init(const ArnState &a, const CycleInit &ci, cudaStream_t s) {
    static_assert(kMaxBatch <= 32 && kArnFlags <= 32, "one warp");
    cycle_init_kernel<<<1, 32, 0, s>>>(a, ci);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_norm2(const VecBatch &x, int R, int nx, int ny, int nz, const int *box, const Reduce &red, double2 *out,
                 long sOut, cudaStream_t s) {
    if (R > red.rmax) return HELM3D_ERR_ARG;
    NormK a = {};
    a.x = x.p;
    a.sX = x.stride;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    if (box) {
        a.phys = 1;
        for (int q = 0; q < 6; q++) a.box[q] = box[q];
    }
    a.partials = red.partials;
    a.sPart = red.stride;
    a.tickets = red.tickets;
    a.out = out;
    a.sOut = sOut;
    const int nb = pass_blocks(red, (long)ny * nz, kRedWarps);
    norm2_kernel<<<dim3(nb, R), kRedThreads, 0, s>>>(a);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_axpby(double2 a, const VecBatch &x, double2 b, const VecBatch &y, long N, int R, cudaStream_t s) {
    axpby_kernel<<<dim3(grid_for(N, R), R), kRedThreads, 0, s>>>(a, x.p, x.stride, b, y.p, y.stride, N);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_sub_dl(const double2 *x, const double2 *dl, const double2 *t, double2 *y, long N, cudaStream_t s) {
    sub_dl_kernel<<<grid_for(N), kRedThreads, 0, s>>>(x, dl, t, y, N);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_set_scale(const double2 *nrm, long sNrm, double *vs, long sVs, int j, int R, cudaStream_t s) {
    set_scale_kernel<<<1, 32 * ((R + 31) / 32), 0, s>>>(nrm, sNrm, vs, sVs, j, R);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

int launch_base2d(bool c64, const double *s2, int nz, long plane, int zlo, int zhi, double w2, double beta,
                  void *base2d, int *status, cudaStream_t s) {
    const unsigned grid = (unsigned)((plane + 255) / 256);
    if (c64) base2d_kernel<float><<<grid, 256, 0, s>>>(s2, nz, plane, zlo, zhi, w2, beta, (float2 *)base2d, status);
    else base2d_kernel<double><<<grid, 256, 0, s>>>(s2, nz, plane, zlo, zhi, w2, beta, (double2 *)base2d, status);
    return ok() ? HELM3D_OK : HELM3D_ERR_CUDA;
}

Dev &device_info() {
    static Dev d;
    static bool init = false;
    if (!init) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceProp p;
        if (cudaGetDeviceProperties(&p, dev) == cudaSuccess) {
            d.sm_count = p.multiProcessorCount;
            d.smem_optin = p.sharedMemPerBlockOptin;
        }
        init = true;
    }
    return d;
}

}  // namespace h3d
