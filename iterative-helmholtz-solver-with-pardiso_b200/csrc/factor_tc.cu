// factor_tc.cu -- the block-tridiagonal factor of blocklu.cu for complex64
// blocks of n <= 128 with the block resident in tensor memory and the
// Gauss-Jordan elimination blocked by panels of 16 columns, the trailing
// updates on the 5th-generation tensor cores (tcgen05, kind::tf32, 3xTF32).
// Same recurrence (replacing PARDISO phases 11/22, Source/FGMRES.cpp:274-284,
// and DirFactFastDiagStructOnline, Source/HODLR/BinaryTreesHODLR.cpp:
// 2870-2969), from both ends towards the middle line (chain.cuh: one launch
// for the halves, one for the middle lines): S_0 = D_0, S_j = D_j - cin[j]
// cout[prev] G_prev, G_j = S_j^{-1}, by Gauss-Jordan with partial pivoting
// (the pivot of column k is the row, among those not yet pivoted, with the
// largest |re| + |im|; ties to the lowest row), G_j^T written row-major for
// the sweep.
//
// Blocking.  Step k of in-place Gauss-Jordan changes every column j != k by
// M[:, j] -= c_k p_k[j] with c_k the current column k (its pivot entry minus
// one) and p_k the normalized pivot row, so the 16 steps of a panel act on
// the columns outside it as M_J <- M_J + X M_J[R, :], R the panel's pivot
// rows and X = (the panel's columns after its 16 steps) - E_R (E_R: ones
// at (r_k, k)).  The panel's steps run on CUDA cores with the panel in
// registers (thread i = row i).
//
// Look-ahead.  The chain of pivot steps bounds the factor, so the four row warps
// do only what the next step needs: they gather the pivot rows' entries in the
// next panel's columns, build their B, issue their GEMM and run that panel's
// steps.  Four helper warps meanwhile gather the other columns (a panel's at a
// time through two small buffers), build B and issue X M[R, :] for every column
// outside panels p and p + 1 (M = 128 rows, K = 32 real), accumulated into the
// block in TMEM, which the row warps wait for only before they write the next X.
// A panel's own columns, which the product does not describe, are rewritten
// from registers.  All columns by the same 3xTF32 product: the next panel's in
// FP32 was no slower, but raised the preconditioner's error at 96^3 from 2.16e-6
// to 2.98e-6.
//
// Frames.  The block is never unscrambled: physical row t of M holds logical
// row rho[t], physical column q logical column kap[q], and the next line's S
// is formed in place in the frame that the pivots leave (the derivation stands
// in factor_tc2.cu).
//
// Layout per CTA (one CTA per (kz, half), its lines in sequence):
//   TMEM (256 columns, lane t = row t): the block (columns 2j / 2j + 1 = Re /
//     Im of column j);
//   shared memory: X (A of the GEMM) and B = real form of M[R, :] (hi and lo,
//     canonical no-swizzle K-major, 128 and 2 ncol rows x 32); the pivot rows
//     in the next panel's columns; the per-warp pivot keys and rows (double-
//     buffered by step parity, so one barrier per step); the frame and the
//     pivot order.  Half of TMEM and of shared memory: two CTAs share an SM.
// Two chains on an SM hide each other's latencies, which is why X is in shared
// memory and not in TMEM (96^3 2.95 ms, 128^3 5.85; one CTA per SM with a whole
// GEMM after each panel and the block unscrambled 5.13, 9.66).
// Every wait is bounded: on expiry bit 1 of *status is set and the kernel
// runs on without waiting (results invalid), waits (bounded) for its MMAs,
// frees its TMEM and returns.  A zero pivot, or a column without a finite
// candidate, sets bit 0.
#include <cuda_runtime.h>

#include <cstdint>

#include "factor_tc.cuh"

namespace h3d {

constexpr int kFtNP = 128;              // rows = TMEM lanes, padded columns
constexpr int kFtYld = kFtB + 2;        // row of Y: reads of four rows at a column fall on distinct banks
constexpr uint32_t kFtCols = 2 * kFtNP; // TMEM columns: two CTAs per SM

struct FtSmem {
    float *Bhi, *Blo;   // [2 kFtNP rows][2 kFtB] canonical each
    float *Xhi, *Xlo;   // [kFtNP rows][2 kFtB] canonical each
    float2 *Yn;         // [kFtB][kFtYld]: the pivot rows in the next panel's columns (the row warps')
    float2 *Y;          // [2][kFtB][kFtYld]: ... in one panel's columns, by turns (the helpers')
    float2 *wrow;       // [2][4][kFtB]
    uint32_t *ckey;     // [2][4]: each warp's pivot key, by step parity
    int *rho, *kap;     // [2][kFtNP] each: the frame, double-buffered by line
    int *kapinv, *perm, *stepof;   // [kFtNP]; stepof[t]: the step that pivoted row t
    uint64_t *x_ready, *next_done, *rest_done, *fin;
    uint32_t *tslot;
};

constexpr size_t kFtSmemBytes = 2 * sizeof(float) * 3 * kFtNP * 2 * kFtB + sizeof(float2) * 3 * kFtB * kFtYld +
                                sizeof(float2) * 2 * 4 * kFtB + sizeof(uint32_t) * 8 + sizeof(int) * 7 * kFtNP +
                                4 * sizeof(uint64_t) + 16;

__device__ __forceinline__ FtSmem ft_carve(unsigned char *raw) {
    FtSmem s;
    s.Bhi = reinterpret_cast<float *>(raw);                       // 1024-aligned base
    s.Blo = s.Bhi + 2 * kFtNP * 2 * kFtB;
    s.Xhi = s.Blo + 2 * kFtNP * 2 * kFtB;
    s.Xlo = s.Xhi + kFtNP * 2 * kFtB;
    s.Yn = reinterpret_cast<float2 *>(s.Xlo + kFtNP * 2 * kFtB);
    s.Y = s.Yn + kFtB * kFtYld;
    s.wrow = s.Y + 2 * kFtB * kFtYld;
    s.ckey = reinterpret_cast<uint32_t *>(s.wrow + 2 * 4 * kFtB);
    s.rho = reinterpret_cast<int *>(s.ckey + 8);
    s.kap = s.rho + 2 * kFtNP;
    s.kapinv = s.kap + 2 * kFtNP;
    s.perm = s.kapinv + kFtNP;
    s.stepof = s.perm + kFtNP;
    s.x_ready = reinterpret_cast<uint64_t *>(s.stepof + kFtNP);   // (every part a multiple of 16 bytes)
    s.next_done = s.x_ready + 1;
    s.rest_done = s.x_ready + 2;
    s.fin = s.x_ready + 3;
    s.tslot = reinterpret_cast<uint32_t *>(s.x_ready + 4);
    return s;
}

// MID: the middle lines (one launch) instead of the halves: a kernel of its
// own, so that the halves' loop does not carry the middle line's code
template <bool MID>
__global__ void __launch_bounds__(kFtThreads, 2) factor_tc_kernel(FtK a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    FtSmem sm = ft_carve(smem_raw);
    const int n = a.n;
    const int kz = MID ? blockIdx.x : blockIdx.x >> 1;
    const HalfChain hc(a.ny, MID ? 0 : blockIdx.x & 1);
    const int lines = MID ? 1 : hc.K;
    const float2 *cin = hc.half ? a.cpy : a.cmy, *cout = hc.half ? a.cmy : a.cpy;
    if (a.kzslot && a.kzslot[kz] >= 0) return;   // a skipped mode (kz_skip_ratio): not factored / swept
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int npan = (n + kFtB - 1) / kFtB;
    const int ncol = npan * kFtB;

    if (warp == 0) tmem_alloc(sm.tslot, kFtCols);
    for (int q = tid; q < kFtNP; q += kFtThreads) {
        sm.rho[q] = sm.rho[kFtNP + q] = q;
        sm.kap[q] = sm.kap[kFtNP + q] = q;
        sm.kapinv[q] = q;
        sm.perm[q] = 0;
        sm.stepof[q] = -1;   // not pivoted in this line yet
    }
    if (tid == 0) {
        mbar_init(sm.x_ready, kFtRowWarps);
        mbar_init(sm.next_done, 1);
        mbar_init(sm.rest_done, 1);
        mbar_init(sm.fin, 1);
        fence_mbar_init_cluster();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *sm.tslot;
    bool dead = false;
    auto wait = [&](uint64_t *bar, uint32_t parity) {   // whole warps
        if (!dead && !mbar_wait_warp_cta(smem_u32(bar), parity, kFtWaitLimit)) {
            dead = true;
            if (lane == 0) atomicOr(a.status, 2);
        }
    };
    const int t = tid & (kFtRowThreads - 1);      // row t, TMEM lane t
    const bool valid = t < n;
    const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const float2 kzv = a.kz2[kz];
    const bool helper = warp >= kFtRowWarps;
    int cur = 0;

    // every other 16-column chunk of the block by each kind of warp, here and
    // at the end of a line
    if (lines > 0) ft_first_block<MID>(a, trow, valid, t, kz, MID ? hc.mid : hc.line(0), ncol, helper ? 1 : 0, kzv);
    tc_fence_before();
    ft_all_barrier();
    tc_fence_after();
    auto line_out = [&](int ls, int which) {
        const int line = MID ? hc.mid : hc.line(ls);
        const bool more = ls + 1 < lines;
        const int nl = more ? hc.line(ls + 1) : 0;
        ft_line_out(a, trow, valid, valid ? sm.rho[cur * kFtNP + t] : 0, sm.kap + cur * kFtNP, sm.kapinv,
                    a.Gt + ((long)kz * a.ny + line) * (long)n * a.ldg, ncol, which, more, nl,
                    more ? cmul(cin[nl], cout[line]) : make_float2(0.f, 0.f), kzv);
        tc_fence_before();
        ft_all_barrier();   // the next line's block is in TMEM
        tc_fence_after();
    };

    const uint32_t bhi = smem_u32(sm.Bhi), blo = smem_u32(sm.Blo), xhi = smem_u32(sm.Xhi), xlo = smem_u32(sm.Xlo);
    // D[:, c0 + [0, len)) += X B[c0 + [0, len), :]^T, 3xTF32
    auto issue = [&](int c0, int len) {
        if (len <= 0) return;
        const uint32_t sbo = (uint32_t)(2 * kFtB / 4) * 128u, idesc = umma_idesc_tf32(len);
        const uint32_t boff = (uint32_t)(c0 / 8) * sbo, d = tmem + (uint32_t)c0;
#pragma unroll
        for (int ks = 0; ks < 2 * kFtB / 8; ks++) {
            const uint32_t koff = (uint32_t)ks * 256u;   // 8 K = two core matrices of 128 B
            const uint64_t dh = umma_desc(bhi + boff + koff, 128, sbo), dl = umma_desc(blo + boff + koff, 128, sbo);
            const uint64_t xh = umma_desc(xhi + koff, 128, sbo), xl = umma_desc(xlo + koff, 128, sbo);
            umma_tf32(d, xh, dh, idesc, 1u);
            umma_tf32(d, xh, dl, idesc, 1u);
            umma_tf32(d, xl, dh, idesc, 1u);
        }
    };

    if (helper) {
        // ------------------------------------------------------- helpers
        const bool issuer = warp == kFtRowWarps && lane == 0;
        uint32_t ph_x = 0, ph_rest = 0;
        for (int ls = 0; ls < lines; ls++) {
            for (int p = 0; p < npan; p++) {
                const int k0 = p * kFtB, bl = min(kFtB, n - k0);
                const int skip = p + 1 < npan ? 2 : 1, nc = npan - skip;
                // the panel's steps are done and its X is in place (the row
                // warps have waited for the previous GEMM)
                wait(sm.x_ready, ph_x);
                ph_x ^= 1u;
                tc_fence_after();
                // ---- the pivot rows (before the panel's update) in the columns
                // outside panels p and p + 1 through Y into B, a panel's columns
                // at a time, the next ones on their way out of TMEM meanwhile
                const int my_step = valid ? sm.stepof[t] : -1;
                const bool piv = my_step >= k0 && my_step < k0 + bl;
                const bool any = __any_sync(0xffffffffu, piv);
                const uint32_t yrow = smem_u32(sm.Y + (piv ? my_step - k0 : 0) * kFtYld);
                const int kk0 = 2 * ((t >> 2) & 7);
                float f[32];
                if (any && nc > 0) tmem_ld32_nowait(trow + (uint32_t)(32 * (p > 0 ? 0 : skip)), f);
#pragma unroll 1
                for (int c = 0; c < nc; c++) {
                    const int cc = c < p ? c : c + skip;
                    const uint32_t half = (uint32_t)((c & 1) * kFtB * kFtYld * sizeof(float2));
                    if (any) {
                        tmem_wait_ld(f);
#pragma unroll
                        for (int e = 0; e < 8; e++)
                            st_shared_v4_if(piv, yrow + half + 16u * (uint32_t)e,
                                            make_float4(f[4 * e], f[4 * e + 1], f[4 * e + 2], f[4 * e + 3]));
                        if (c + 1 < nc) tmem_ld32_nowait(trow + (uint32_t)(32 * (c + 1 < p ? c + 1 : c + 1 + skip)), f);
                    }
                    ft_helper_barrier();
                    const float2 *y = sm.Y + ((c & 1) * kFtB + kk0) * kFtYld + (t >> 5) * 4 + (t & 3);
                    ft_put_b(sm.Bhi, sm.Blo, 128 * cc + t, kk0 < bl ? y[0] : make_float2(0.f, 0.f),
                             kk0 + 1 < bl ? y[kFtYld] : make_float2(0.f, 0.f));
                }
                tc_fence_before();
                fence_proxy_async_smem();
                ft_helper_barrier();
                tc_fence_after();
                if (issuer) {
                    issue(0, 2 * kFtB * p);
                    if (skip == 2) issue(2 * kFtB * (p + 2), 2 * ncol - 2 * kFtB * (p + 2));
                    umma_commit(sm.rest_done);
                }
                __syncwarp();
                if (skip == 2) ph_rest ^= 1u;   // (waited for by the row warps)
            }
            wait(sm.rest_done, ph_rest);
            ph_rest ^= 1u;
            tc_fence_after();
            ft_all_barrier();   // the next frame
            cur ^= 1;
            line_out(ls, 1);
        }
        if (issuer) {
            umma_commit(sm.fin);
            mbar_wait_bounded_cta(smem_u32(sm.fin), 0u, kFtWaitLimit);
        }
        __syncwarp();
    } else {
        // ----------------------------------------------------- row threads
        uint32_t ph_rest = 0, ph_next = 0;
        for (int ls = 0; ls < lines; ls++) {
            bool used = false;
            int my_step = -1;
            float2 P[kFtB];
            {   // the first panel's columns
                float f[32];
                tmem_ld32_nowait(trow, f);
                tmem_wait_ld(f);
#pragma unroll
                for (int e = 0; e < kFtB; e++) P[e] = make_float2(f[2 * e], f[2 * e + 1]);
            }
            for (int p = 0; p < npan; p++) {
                const int k0 = p * kFtB, bl = min(kFtB, n - k0);
                // ---- the panel's steps (CUDA cores), in a rolled loop: the row
                // rotates by one column per step, so that the column of step kk
                // is always P[0]; after step kk, P[e] holds panel column
                // (kk + 1 + e) mod 16.  The pivot of a column is the candidate
                // row with the largest key: the top 24 bits of |re| + |im| and
                // 255 - row (ties, to 2^-15 relative, go to the lowest row),
                // reduced per warp by redux.sync and across the 4 warps through
                // shared memory slots alternating by step parity.  The pivot
                // row keeps its values in its step (multiplier 0, new column 1)
                // and is scaled by its 1 / pv after the panel: every later step
                // is linear in the row.  The next step's warp reduction is
                // issued right after the update of the next pivot column.
                float2 psc = make_float2(1.f, 0.f);
                bool pivp = false, bad = false;
                uint32_t key = 0;
                {
                    const float av = fabsf(P[0].x) + fabsf(P[0].y);
                    if (!used && t < n && av == av) key = (__float_as_uint(av) & 0xFFFFFF00u) | (uint32_t)(255 - t);
                }
                uint32_t kw = __reduce_max_sync(0xffffffffu, key);
#pragma unroll 1
                for (int kk = 0; kk < bl; kk++) {
                    const int k = k0 + kk, buf = k & 1;
                    st_shared_u32_if(lane == 0, smem_u32(&sm.ckey[buf * 4 + warp]), kw);
                    {
                        // the winning row in register order: w[0] the pivot, w[1 + e] = prow[e]
                        const bool win = kw != 0u && key == kw;
                        const uint32_t w = smem_u32(sm.wrow + (buf * 4 + warp) * kFtB);
#pragma unroll
                        for (int e = 0; e < kFtB / 2; e++)
                            st_shared_v4_if(win, w + 16u * (uint32_t)e,
                                            make_float4(P[2 * e].x, P[2 * e].y, P[2 * e + 1].x, P[2 * e + 1].y));
                    }
                    ft_row_barrier();
                    const uint4 kv = *reinterpret_cast<const uint4 *>(sm.ckey + buf * 4);
                    uint32_t kmax = kv.x;
                    int wsel = 0;
                    if (kv.y > kmax) {
                        kmax = kv.y;
                        wsel = 1;
                    }
                    if (kv.z > kmax) {
                        kmax = kv.z;
                        wsel = 2;
                    }
                    if (kv.w > kmax) {
                        kmax = kv.w;
                        wsel = 3;
                    }
                    const int r = kmax != 0u ? 255 - (int)(kmax & 0xFFu) : -1;
                    // the pivot row, rotated like the rows: prow[e] = column (kk + 1 + e) mod 16
                    const float4 *w = reinterpret_cast<const float4 *>(sm.wrow + (buf * 4 + wsel) * kFtB);
                    float2 prow[kFtB], pv = make_float2(0.f, 0.f);
#pragma unroll
                    for (int e = 0; e < kFtB / 2; e++) {
                        const float4 q4 = w[e];
                        if (e == 0) pv = make_float2(q4.x, q4.y);
                        else prow[2 * e - 1] = make_float2(q4.x, q4.y);
                        prow[2 * e] = make_float2(q4.z, q4.w);
                    }
                    // no finite candidate, or an exactly zero pivot: flagged (after
                    // the panel), the block is invalid
                    const bool none = r < 0 || (pv.x == 0.f && pv.y == 0.f);
                    bad |= none;
                    const float2 pi = pivot_inv(pv);
                    const float2 pinv = make_float2(none ? 0.f : pi.x, none ? 0.f : pi.y);
                    // row -= (c / pv) * pivot row, column k becomes -c / pv
                    const bool ip = t == r;
                    float2 sfac = cmul(P[0], pinv);
                    sfac = make_float2(ip ? 0.f : sfac.x, ip ? 0.f : sfac.y);
                    psc = make_float2(ip ? pinv.x : psc.x, ip ? pinv.y : psc.y);
                    used |= ip;
                    pivp |= ip;
                    my_step = ip ? k : my_step;
                    st_shared_u32_if(ip, smem_u32(&sm.perm[k]), (uint32_t)t);
                    st_shared_u32_if(ip, smem_u32(&sm.stepof[t]), (uint32_t)k);
                    P[0] = cfms(sfac, prow[0], P[1]);
                    key = 0;
                    {
                        const float av = fabsf(P[0].x) + fabsf(P[0].y);
                        if (!used && t < n && av == av) key = (__float_as_uint(av) & 0xFFFFFF00u) | (uint32_t)(255 - t);
                    }
                    kw = __reduce_max_sync(0xffffffffu, key);
#pragma unroll
                    for (int e = 1; e < kFtB - 1; e++) P[e] = cfms(sfac, prow[e], P[e + 1]);
                    P[kFtB - 1] = ip ? make_float2(1.f, 0.f) : make_float2(-sfac.x, -sfac.y);
                }
                if (bad && t == 0) atomicOr(a.status, 1);
                // the panel's pivot row scaled by its 1 / pv
                if (pivp) {
#pragma unroll
                    for (int e = 0; e < kFtB; e++) P[e] = cmul(P[e], psc);
                }
                // back to column order (P[e] holds column (bl + e) mod 16; only
                // a partial last panel is not back in order): rotated by bl
#pragma unroll
                for (int b = 1; b < kFtB; b *= 2)
                    if (bl & b) {
                        float2 Q[kFtB];
#pragma unroll
                        for (int e = 0; e < kFtB; e++) Q[(e + b) & (kFtB - 1)] = P[e];
#pragma unroll
                        for (int e = 0; e < kFtB; e++) P[e] = Q[e];
                    }

                // ---- the previous panel's GEMM is done: X = panel - E_R into
                // shared memory (tf32 hi / lo), the panel's own columns into TMEM,
                // the next panel's columns out of it
                if (p > 0) {
                    wait(sm.rest_done, ph_rest);
                    ph_rest ^= 1u;
                    tc_fence_after();
                }
                const bool next = p + 1 < npan;
                {
                    float f[32];
#pragma unroll
                    for (int e = 0; e < kFtB; e++) {
                        f[2 * e] = P[e].x;
                        f[2 * e + 1] = P[e].y;
                    }
                    tmem_st32(trow + (uint32_t)(2 * k0), f);
                    float *xh = sm.Xhi + canon_off(t, 0, 2 * kFtB) / 4, *xl = sm.Xlo + canon_off(t, 0, 2 * kFtB) / 4;
#pragma unroll
                    for (int e = 0; e < kFtB; e += 2) {
#pragma unroll
                        for (int h = e; h < e + 2; h++) {   // P becomes X
                            P[h].x = h >= bl ? 0.f : my_step == k0 + h ? P[h].x - 1.f : P[h].x;
                            P[h].y = h >= bl ? 0.f : P[h].y;
                        }
                        float4 h4, l4;
                        tf32_split_fast(P[e].x, h4.x, l4.x);
                        tf32_split_fast(P[e].y, h4.y, l4.y);
                        tf32_split_fast(P[e + 1].x, h4.z, l4.z);
                        tf32_split_fast(P[e + 1].y, h4.w, l4.w);
                        *reinterpret_cast<float4 *>(xh + 16 * e) = h4;
                        *reinterpret_cast<float4 *>(xl + 16 * e) = l4;
                    }
                }
                fence_proxy_async_smem();
                float m[32];
                if (next) {
                    tmem_ld32_nowait(trow + (uint32_t)(32 * (p + 1)), m);
                    tmem_wait_ld(m);
                }
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive_warp(sm.x_ready);
                if (!next) break;
                // ---- the next panel's columns: their pivot entries, B (one unit per
                // thread) and GEMM by the row warps, which wait for nothing else
                {
                    const uint32_t yrow = smem_u32(sm.Yn + (pivp ? my_step - k0 : 0) * kFtYld);
#pragma unroll
                    for (int e = 0; e < 8; e++)
                        st_shared_v4_if(pivp, yrow + 16u * (uint32_t)e,
                                        make_float4(m[4 * e], m[4 * e + 1], m[4 * e + 2], m[4 * e + 3]));
                }
                ft_row_barrier();
                {
                    const float2 *y = sm.Yn + 2 * ((t >> 2) & 7) * kFtYld + (t >> 5) * 4 + (t & 3);
                    ft_put_b(sm.Bhi, sm.Blo, 128 * (p + 1) + t, y[0], y[kFtYld]);
                }
                fence_proxy_async_smem();
                tc_fence_before();
                ft_row_barrier();
                tc_fence_after();
                if (t == 0) {
                    issue(2 * kFtB * (p + 1), 2 * kFtB);
                    umma_commit(sm.next_done);
                }
                __syncwarp();
                wait(sm.next_done, ph_next);
                ph_next ^= 1u;
                tc_fence_after();
                tmem_ld32_nowait(trow + (uint32_t)(32 * (p + 1)), m);
                tmem_wait_ld(m);
#pragma unroll
                for (int e = 0; e < kFtB; e++) P[e] = make_float2(m[2 * e], m[2 * e + 1]);
            }

            // ---- the line's last GEMM done: the next frame, G_line^T to global
            // memory and S_{line+1} in place
            wait(sm.rest_done, ph_rest);
            ph_rest ^= 1u;
            tc_fence_after();
            ft_row_barrier();
            const int nxt = cur ^ 1;
            ft_next_frame(n, t, sm.rho + cur * kFtNP, sm.kap + cur * kFtNP, sm.rho + nxt * kFtNP, sm.kap + nxt * kFtNP,
                          sm.kapinv, sm.perm, sm.stepof);
            ft_all_barrier();
            cur = nxt;
            line_out(ls, 0);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kFtCols);
}

bool factor_tc_supported(bool c64, int n) { return c64 && n >= 1 && n <= kFtNP; }

int launch_factor_tc(const FactorArgs &fa, cudaStream_t st) {
    if (fa.n < 1 || fa.n > kFtNP) return HELM3D_ERR_ARG;
    if (kFtSmemBytes > device_info().smem_optin) return HELM3D_ERR_ARG;
    void (*kern)(FtK) = fa.middle ? factor_tc_kernel<true> : factor_tc_kernel<false>;
    if (!smem_limit_max(kern, kFtSmemBytes)) return HELM3D_ERR_CUDA;
    kern<<<dim3((unsigned)((fa.middle ? 1 : 2) * fa.nz)), kFtThreads, kFtSmemBytes, st>>>(ft_args(fa));
    return cudaGetLastError() == cudaSuccess ? HELM3D_OK : HELM3D_ERR_CUDA;
}

}  // namespace h3d
