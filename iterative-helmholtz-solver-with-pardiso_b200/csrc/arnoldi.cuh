// arnoldi.cuh -- the per-step bookkeeping of the lockstep batched FGMRES on
// the device: the Gram-Schmidt second-pass test, the Givens update of the
// Hessenberg column and the right-hand side g, the convergence estimate, and
// the back substitution y = R^{-1} g at the end of a cycle, for one right-hand
// side p by one warp.  The arithmetic is the host loop's (FGMRES restart cycle,
// Source/FGMRES.cpp:464-684, with Givens rotations in place of the per-step
// zgels), in FP64.
//
// It runs at the end of the reduction and update passes (krylov.cu), in the
// block that finishes last: a kernel of its own for each piece, one thread per
// right-hand side, took 2.7-13 us a step (38 us for the back substitution)
// where a step's passes over a 64^3 basis take 46.  The columns are staged in
// shared memory (scr), the sums and products spread over the lanes; only the
// chain of earlier rotations is serial, in lane 0.
//
// A whole restart cycle runs as one CUDA graph: the update pass of step j
// decides, on the device, whether step j + 1 runs (graph conditional node) --
// it runs while some right-hand side of the batch has not converged, reached
// the iteration limit or broken down.
#pragma once
#include "cplx.cuh"
#include "helm3d_internal.h"

namespace h3d {

__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cmag(double2 a) { return hypot(a.x, a.y); }
__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    }
    return v;
}

// double2 values of shared scratch that a step-j bookkeeping takes: the dots
// (2 j + 2), the column (j + 2) and the earlier rotations (2 j)
__host__ __device__ constexpr size_t arn_scratch(int j) { return (size_t)5 * j + 8; }

// Column j (shared memory, unrotated: V^H w above the diagonal, col[j + 1]
// below it): apply the earlier rotations, make rotation j, update g, the
// iteration count and the estimate, store the column to H; returns whether
// right-hand side p stops (converged, iteration limit, breakdown or
// non-finite), the same in every lane.
__device__ inline bool finalize_column(const ArnState &a, int p, int j, double2 *col, double2 *rot) {
    const int m = a.m, lane = threadIdx.x & 31;
    double2 *H = a.H + (long)p * (m + 1) * m;
    double2 *cs = a.cs + (long)p * m, *sn = a.sn + (long)p * m, *g = a.g + (long)p * (m + 1);
    double2 *scs = rot, *ssn = rot + j;
    const double2 gj = g[j];
    const double nf = a.nf[p], tol = a.tol[p];
    const int it = a.it[p] + 1, max_iter = a.max_iter[p];
    for (int i = lane; i < j; i += 32) {
        scs[i] = cs[i];
        ssn[i] = sn[i];
    }
    __syncwarp();
    int frozen = 0;
    if (lane == 0) {
        const double hn = cmag(col[j + 1]);
        double2 x = col[0];
        for (int i = 0; i < j; i++) {
            const double2 y = col[i + 1], c = scs[i], s = ssn[i];
            col[i] = cadd(cmul(c, x), cmul(s, y));
            x = csub(cmul(c, y), cmul(cconj(s), x));
        }
        const double2 y = col[j + 1];
        const double ax = cmag(x), den = hypot(ax, cmag(y));
        double2 c, s;
        if (den == 0.0) {
            c = make_double2(1, 0);
            s = make_double2(0, 0);
        } else if (ax == 0.0) {
            c = make_double2(0, 0);
            s = make_double2(1, 0);
        } else {
            c = make_double2(ax / den, 0.0);
            // (x / |x|) conj(y) / den
            s = cmul(make_double2(x.x / ax, x.y / ax), cconj(y));
            s = make_double2(s.x / den, s.y / den);
        }
        cs[j] = c;
        sn[j] = s;
        col[j] = cadd(cmul(c, x), cmul(s, y));
        col[j + 1] = make_double2(0, 0);
        const double2 gn = make_double2(-(s.x * gj.x + s.y * gj.y), -(s.x * gj.y - s.y * gj.x));   // -conj(s) g[j]
        g[j + 1] = gn;
        g[j] = cmul(c, gj);
        a.it[p] = it;
        a.k[p] = j + 1;
        const double est = cmag(gn) / nf;
        a.est[(long)p * m + j] = est;
        const bool bad = !isfinite(hn) || !isfinite(est);
        if (bad) atomicOr(&a.flags[3], 1);
        frozen = bad || hn == 0.0 || est <= tol || it >= max_iter;
        a.frozen[p] = frozen;
    }
    __syncwarp();
    for (int i = lane; i <= j + 1; i += 32) H[(long)i * m + j] = col[i];
    return __shfl_sync(0xffffffffu, frozen, 0) != 0;
}

// Classical Gram-Schmidt (mode R, or HELM3D_GS=cgs2): the end of step j for
// right-hand side p, h1 (+ h2 after a second pass) and ||w||^2 in a.h.
// Returns whether p goes on.
__device__ inline bool givens_step(const ArnState &a, int p, int j, double2 *scr) {
    const int lane = threadIdx.x & 31;
    double *vs = a.vs + (long)p * a.M2;
    // a right-hand side that has stopped gets zero scales: its further basis
    // vectors are exact zeros (the zero-padded combine then adds nothing)
    if (a.frozen[p]) {
        if (lane == 0) vs[j + 1] = 0.0;
        return false;
    }
    const double2 *h1 = a.h + (long)p * a.SH, *h2 = h1 + a.M2;
    const bool second = a.flags[0] != 0;
    const double hn = sqrt(fmax(0.0, h1[2 * a.M2].x));
    double2 *col = scr, *rot = scr + j + 2;
    for (int i = lane; i <= j; i += 32) col[i] = second ? cadd(h1[i], h2[i]) : h1[i];
    if (lane == 0) col[j + 1] = make_double2(hn, 0.0);
    __syncwarp();
    const bool frozen = finalize_column(a, p, j, col, rot);
    if (lane == 0) vs[j + 1] = (!frozen && hn > 0.0) ? 1.0 / hn : 0.0;
    return !frozen;
}

// ------------------------------------------------ DCGS2 (mode N, flexible)
// Step j computed w = A z_j with z_j = M^{-1} (vs_j V_j), where V_j is still
// the tentative vector of step j - 1 (projected once).  From the one
// reduction pass (val: b_i = vs_i <V_i, w> for i <= j, a_i = vs_i <V_i, V_j>
// for i < j, g = <V_j, V_j>) this
//   * reorthogonalizes V_j: s_i = a_i vs_j, nrm^2 = g vs_j^2 - sum |s_i|^2;
//   * finalizes column j - 1, whose subdiagonal was left open: with
//     beta = ||w_{j-1}'|| of the last update, H[i][j-1] += beta s_i and
//     H[j][j-1] = beta nrm, then its Givens rotation (convergence is known
//     one step late);
//   * writes column j (unrotated) against the final basis: c_i = b_i (i < j),
//     c_j = (b_j - sum conj(s_i) b_i) / nrm;
//   * writes the update coefficients in stored-vector terms (alpha for V_j,
//     delta for w) and the new scale of V_j.
// Frozen right-hand sides are skipped by the passes that follow.
__device__ inline void lagged_step(const ArnState &a, int p, int j, const double2 *val, double2 *scr) {
    const int m = a.m, M2 = a.M2, lane = threadIdx.x & 31;
    double2 *hp = a.h + (long)p * a.SH;
    const double2 *b = val, *av = val + j + 1;
    double2 *alpha = hp + 4 * M2, *delta = hp + 5 * M2;
    double *vs = a.vs + (long)p * M2;
    double2 *H = a.H + (long)p * (m + 1) * m;
    const double sj = vs[j];
    double nrm = 1.0;
    double2 cj = b[j];
    if (j > 0) {
        double2 *col = scr, *rot = scr + j + 1;
        const double beta = a.beta[p];
        double2 ss = make_double2(0, 0), sb = make_double2(0, 0);
        for (int i = lane; i < j; i += 32) {
            const double2 si = cscale(av[i], sj);
            ss.x += si.x * si.x + si.y * si.y;
            sb = cadd(sb, cmul(cconj(si), b[i]));
            col[i] = cadd(H[(long)i * m + j - 1], cscale(si, beta));
        }
        ss = warp_sum(ss);
        sb = warp_sum(sb);
        const double n2 = val[2 * j + 1].x * sj * sj - ss.x;
        nrm = n2 > 0.0 ? sqrt(n2) : 0.0;
        if (lane == 0) col[j] = make_double2(beta * nrm, 0.0);
        __syncwarp();
        if (finalize_column(a, p, j - 1, col, rot)) return;
        cj = csub(cj, sb);
    }
    // nrm > 0 here: nrm = 0 makes H[j][j-1] = 0, a breakdown that stops p
    cj = cscale(cj, 1.0 / nrm);
    const double2 cn = cscale(cj, 1.0 / nrm);
    for (int i = lane; i < j; i += 32) {
        H[(long)i * m + j] = b[i];
        const double2 si = cscale(av[i], sj);
        alpha[i] = cscale(si, vs[i] / sj);
        delta[i] = cscale(csub(b[i], cmul(cn, si)), vs[i]);
    }
    __syncwarp();
    if (lane == 0) {
        H[(long)j * m + j] = cj;
        delta[j] = cscale(cj, sj / nrm);
        if (j > 0) vs[j] = sj / nrm;
    }
}

// After the update pass of step j: beta = ||w'||, the scale of the new
// tentative vector V_{j+1}, the breakdown and non-finite checks; one thread.
// Returns whether p goes on.
__device__ inline bool post_step(const ArnState &a, int p, int j, double norm2) {
    double *vs = a.vs + (long)p * a.M2;
    if (a.frozen[p]) {
        vs[j + 1] = 0.0;
        return false;
    }
    const double beta = sqrt(fmax(0.0, norm2));
    if (!isfinite(beta)) {
        atomicOr(&a.flags[3], 1);
        a.frozen[p] = 1;
        vs[j + 1] = 0.0;
        return false;
    }
    a.beta[p] = beta;
    vs[j + 1] = beta > 0.0 ? 1.0 / beta : 0.0;
    return true;
}

// End of a cycle: the open column jl = t - 1 of a still active right-hand
// side, from the reorthogonalization dots of V_t (val: a_i at 0 .. jl, g at t).
__device__ inline void lagged_final(const ArnState &a, int p, int t, const double2 *val, double2 *scr) {
    const int m = a.m, jl = t - 1, lane = threadIdx.x & 31;
    const double st = a.vs[(long)p * a.M2 + t], beta = a.beta[p];
    double2 *H = a.H + (long)p * (m + 1) * m;
    double2 *col = scr, *rot = scr + t + 1;
    double2 ss = make_double2(0, 0);
    for (int i = lane; i <= jl; i += 32) {
        const double2 si = cscale(val[i], st);
        ss.x += si.x * si.x + si.y * si.y;
        col[i] = cadd(H[(long)i * m + jl], cscale(si, beta));
    }
    ss = warp_sum(ss);
    const double n2 = val[t].x * st * st - ss.x;
    const double nrm = n2 > 0.0 ? sqrt(n2) : 0.0;
    if (lane == 0) col[t] = make_double2(beta * nrm, 0.0);
    __syncwarp();
    finalize_column(a, p, jl, col, rot);
    if (lane == 0) a.frozen[p] = 1;
}

// y = R^{-1} g for right-hand side p by a whole block: columns from the last
// to the first, each lane of warp 0 updating its entries of g (shared memory);
// the triangle staged in shared memory (tri) up to kBacksubTri columns.
constexpr int kBacksubTri = 32;
__device__ inline void backsub_block(const ArnState &a, int p, double2 *gs, double2 *tri) {
    const int m = a.m, k = a.k[p];
    const double2 *H = a.H + (long)p * (m + 1) * m, *g = a.g + (long)p * (m + 1);
    double2 *y = a.h + (long)p * a.SH + 3 * a.M2;
    const bool staged = k <= kBacksubTri;
    for (int i = threadIdx.x; i < k; i += blockDim.x) gs[i] = g[i];
    if (staged)
        for (int q = threadIdx.x; q < k * k; q += blockDim.x) tri[q] = H[(long)(q / k) * m + q % k];
    for (int i = k + threadIdx.x; i < m; i += blockDim.x) y[i] = make_double2(0, 0);
    __syncthreads();
    if (threadIdx.x < 32) {
        for (int i = k - 1; i >= 0; i--) {
            const double2 yi = cmul(gs[i], cinv(staged ? tri[i * k + i] : H[(long)i * m + i]));
            if (threadIdx.x == 0) y[i] = yi;
            for (int q = threadIdx.x; q < i; q += 32)
                gs[q] = csub(gs[q], cmul(staged ? tri[q * k + i] : H[(long)q * m + i], yi));
            __syncwarp();
        }
    }
}

}  // namespace h3d
