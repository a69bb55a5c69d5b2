// factor_tc2.cu -- the block-tridiagonal factor of blocklu.cu for complex64
// blocks of 128 < n <= 224 on a pair of CTAs per (kz, half) (a thread-block cluster
// of 2), the block resident in the two CTAs' tensor memory and the trailing
// updates of the panel-blocked Gauss-Jordan elimination on the tensor cores
// (tcgen05, kind::tf32, 3xTF32).  Same recurrence as blocklu.cu and
// factor_tc.cu (replacing PARDISO phases 11/22, Source/FGMRES.cpp:274-284, and
// DirFactFastDiagStructOnline, Source/HODLR/BinaryTreesHODLR.cpp:2870-2969):
// from both ends towards the middle line (chain.cuh: one launch for the
// halves, one for the middle lines),
// S_0 = D_0, S_j = D_j - cin[j] cout[prev] G_prev, G_j = S_j^{-1}, by
// Gauss-Jordan with partial pivoting, G_j^T written row-major for the sweep.
//
// Rows.  CTA 0 of the pair holds physical rows [0, n0), CTA 1 rows [n0, n)
// (n0 = ceil(n/2) <= 112), one row per TMEM lane (lane = row - first row);
// every CTA holds all 2 ncol real columns (ncol = n rounded up to the panel
// width 16): TMEM columns [0, 2 ncol) hold M (2j, 2j+1 = Re, Im of column j),
// [2 ncol, 2 ncol + 32) and [2 ncol + 32, 2 ncol + 64) the panel's X = panel
// - E_R as tf32 hi / lo.  Each CTA runs its own tcgen05 GEMMs (M = 128 rows,
// its own lanes) with its own copy of B (the real form of the panel's pivot
// rows) in shared memory.
//
// Panels.  A panel's 16 pivot steps touch only the panel's columns, n x 16
// complex values, so both CTAs run all of them, on the whole panel, with the
// same arithmetic and therefore the same pivots: at the start of a panel
// each CTA sends its rows' panel entries into both CTAs' shared memory
// (cluster stores, then one arrive per warp on the peer's barrier, release
// at cluster scope), and thread t of each CTA takes physical rows t and
// t + 128 into registers.  A step is then local to the CTA: the pivot
// candidate of each warp is one 32-bit key (redux.sync.max): the top 24
// bits of |re| + |im| and 255 - row, so that the largest magnitude wins and
// ties go to the lowest row (magnitudes equal to 2^-15 relative count as
// ties); the warps' keys and winning rows go through shared memory slots
// alternating by step parity, one CTA barrier per step.  After the steps
// each CTA keeps X and the panel of its own rows, and the panel's pivot
// rows (their other columns live in their owner's TMEM) are exchanged the
// same way as the panel entries.
//
// Frames.  The block is never unscrambled.  Physical row g of M holds
// logical row rho[g], physical column q logical column kap[q].  In-place
// Gauss-Jordan without row exchanges on A[g][q] = S[rho[g]][kap[q]] leaves
// M[g][q] = S^{-1}[kap[sigma[g]]][rho[perm[q]]] with perm[k] the pivot row
// of step k and sigma its inverse (the step of row g), so the next frame is
// rho' = kap o sigma, kap' = rho o perm.  The next Schur complement is
// formed in place in that frame, M <- D[rho'][kap'] - c M (D tridiagonal:
// three entries per row, at the physical columns kapinv of logical columns
// i-1, i, i+1), and G_j^T is written to global memory as
// G^T[kap'[q]][rho'[g]] = M[g][q] (the 8-byte stores of a warp scatter
// within one row of G^T and merge in L2).
//
// Look-ahead.  The chain of pivot steps bounds the factor, so the four row
// warps do only what the next step needs: after panel p's steps they exchange
// its pivot rows in the next panel's 16 columns, build those columns' B and,
// when their GEMM is done (next_ready), run panel p+1's steps.  Four helper
// warps meanwhile exchange the pivot rows' other columns, build their B and
// issue the GEMM of every column outside panels p and p+1 (rest_done), which the
// row warps wait for only before they write panel p+1's X.  A finished line is
// written, and the next one formed, by all eight warps.
//
// 200 x 200 x 74: 39.7 ms by the row warps alone with branches in a step, 29.6 so.
// A step is 725 cycles: store the candidate 130, barrier 25, keys 105, the row 85,
// the next column's update and reduction 180, the other columns 160.  Eight row
// warps of one row each were slower by 5 %: more warps at each barrier.
//
// Tensor memory.  Two kernels whose clusters hold some on one SM while they wait
// for some on another could wait for each other.  The only other cluster kernel
// with tensor memory is the packed sweep (352 threads of at least 80 registers),
// and beside a CTA of this one (256 threads of at least 168) an SM has registers
// for 64 each: the two never share an SM.
//
// Every wait is bounded: on expiry bit 1 of *status is set and the kernel
// runs on without waiting (results invalid), waits (bounded) for its MMAs,
// meets its peer at a final cluster barrier (so that no store into a
// CTA's shared memory can land after it exits), frees its TMEM and returns.
// A zero pivot, or a column without a finite candidate, sets bit 0.
#include <cuda_runtime.h>

#include <cstdint>

#include "factor_tc.cuh"

namespace h3d {

constexpr int kF2MaxN = 224;                     // 2 ncol + 64 X columns <= 512
constexpr int kF2Tab = 256;
constexpr uint32_t kF2Cols = 512;

struct F2Smem {
    float *Bhi, *Blo;   // [2 kF2MaxN rows][2 kFtB] canonical K-major each
    float2 *Y;          // [kFtB][kF2Yld]: the panel's pivot rows (the helpers')
    float2 *Yn;         // [kFtB][kF2PFld]: their entries in the next panel's columns (the row warps')
    float2 *PF;         // [kF2MaxN][kF2PFld]: the panel's entries of every row
    float2 *wrow;       // [2][kFtRowWarps][kFtB]: each warp's candidate row, by step parity
    uint32_t *wkey;     // [2][kFtRowWarps]
    int *rho, *kap;     // [2][kF2Tab] each: the frame, double-buffered by line
    int *kapinv, *perm, *stepof;   // [kF2Tab]; stepof[g]: the step that pivoted row g
    uint64_t *pan_bar, *yn_bar, *bn_ready, *x_ready, *y_bar, *y_free, *next_ready, *rest_done, *fin;
    uint32_t *tslot;
};

constexpr size_t kF2BBytes = sizeof(float) * 2 * kF2MaxN * 2 * kFtB;
// row stride of PF: 18 complex (144 bytes) instead of 16, so that a warp's
// row-per-thread accesses (16-byte and 8-byte) fall on distinct banks
constexpr int kF2PFld = kFtB + 2;
// row stride of Y: 226 complex, so that the B build's reads of four pivot
// rows at the same column fall on distinct banks (16-byte aligned rows)
constexpr int kF2Yld = kF2MaxN + 2;
constexpr size_t kF2SmemBytes = 2 * kF2BBytes + sizeof(float2) * (kFtB * kF2Yld + kFtB * kF2PFld + kF2PFld * kF2MaxN) +
                                sizeof(float2) * 2 * kFtRowWarps * kFtB + sizeof(uint32_t) * 2 * kFtRowWarps +
                                sizeof(int) * 7 * kF2Tab + 9 * sizeof(uint64_t) + 16 + 1024 + 16;

__device__ __forceinline__ F2Smem f2_carve(unsigned char *raw) {
    F2Smem s;
    uintptr_t b = (reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023);
    s.Bhi = reinterpret_cast<float *>(b);
    s.Blo = s.Bhi + 2 * kF2MaxN * 2 * kFtB;
    s.Y = reinterpret_cast<float2 *>(s.Blo + 2 * kF2MaxN * 2 * kFtB);
    s.Yn = s.Y + kFtB * kF2Yld;
    s.PF = s.Yn + kFtB * kF2PFld;
    s.wrow = s.PF + kF2MaxN * kF2PFld;
    s.wkey = reinterpret_cast<uint32_t *>(s.wrow + 2 * kFtRowWarps * kFtB);
    s.rho = reinterpret_cast<int *>(s.wkey + 2 * kFtRowWarps);
    s.kap = s.rho + 2 * kF2Tab;
    s.kapinv = s.kap + 2 * kF2Tab;
    s.perm = s.kapinv + kF2Tab;
    s.stepof = s.perm + kF2Tab;
    uintptr_t m = reinterpret_cast<uintptr_t>(s.stepof + kF2Tab);
    m = (m + 15) & ~uintptr_t(15);
    s.pan_bar = reinterpret_cast<uint64_t *>(m);
    s.yn_bar = s.pan_bar + 1;
    s.bn_ready = s.pan_bar + 2;
    s.x_ready = s.pan_bar + 3;
    s.y_bar = s.pan_bar + 4;
    s.y_free = s.pan_bar + 5;
    s.next_ready = s.pan_bar + 6;
    s.rest_done = s.pan_bar + 7;
    s.fin = s.pan_bar + 8;
    s.tslot = reinterpret_cast<uint32_t *>(s.pan_bar + 9);
    return s;
}

__device__ __forceinline__ void st_cluster_v4f32(uint32_t addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z),
                 "f"(v.w)
                 : "memory");
}

// MID: the middle lines (one launch) instead of the halves: a kernel of its
// own, so that the halves' loop does not carry the middle line's code
template <bool MID>
__global__ void __launch_bounds__(kFtThreads, 1) factor_tc2_kernel(FtK a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    F2Smem sm = f2_carve(smem_raw);
    const int n = a.n;
    const uint32_t rank = blockIdx.x & 1u, peer = rank ^ 1u;   // the rank in the cluster of two
    const int piece = blockIdx.x >> 1;
    const int kz = MID ? piece : piece >> 1;
    const HalfChain hc(a.ny, MID ? 0 : piece & 1);
    const int lines = MID ? 1 : hc.K;
    const float2 *cin = hc.half ? a.cpy : a.cmy, *cout = hc.half ? a.cmy : a.cpy;
    if (a.kzslot && a.kzslot[kz] >= 0) return;   // a skipped mode (kz_skip_ratio): not factored / swept
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
    const int n0 = (n + 1) >> 1;
    const int nr = rank == 0 ? n0 : n - n0;       // rows of this CTA
    const int gbase = rank == 0 ? 0 : n0;
    const int ncol = (n + kFtB - 1) / kFtB * kFtB;
    const int npan = ncol / kFtB;
    const uint32_t kXhi = 2u * ncol, kXlo = 2u * ncol + 32u;

    if (warp == 0) tmem_alloc(sm.tslot, kF2Cols);
    for (int q = tid; q < kF2Tab; q += kFtThreads) {
        sm.rho[q] = q;
        sm.kap[q] = q;
        sm.kapinv[q] = q;
        sm.perm[q] = 0;
        sm.stepof[q] = -1;   // not pivoted in this line yet
    }
    if (tid == 0) {
        mbar_init(sm.pan_bar, kFtRowWarps);   // the peer's row warps
        mbar_init(sm.yn_bar, kFtRowWarps);    // the peer's row warps
        mbar_init(sm.bn_ready, kFtRowWarps);
        mbar_init(sm.x_ready, kFtRowWarps);
        mbar_init(sm.y_bar, kFtRowWarps);     // the peer's helpers
        mbar_init(sm.y_free, kFtRowWarps);    // the peer's helpers
        mbar_init(sm.next_ready, 1);
        mbar_init(sm.rest_done, 1);
        mbar_init(sm.fin, 1);
        fence_mbar_init_cluster();
    }
    tc_fence_before();
    cluster_sync_all();   // both CTAs' barriers exist before any remote arrive
    tc_fence_after();
    const uint32_t tmem = *sm.tslot;
    bool dead = false;
    // waits by whole warps
    auto wait_warp = [&](uint64_t *bar, uint32_t parity) {
        if (!dead && !mbar_wait_warp_cta(smem_u32(bar), parity, kFtWaitLimit)) {
            dead = true;
            atomicOr(a.status, 2);
        }
    };
    auto wait_cluster = [&](uint64_t *bar, uint32_t parity) {
        if (!dead && !mbar_wait_warp_cluster(smem_u32(bar), parity, kFtWaitLimit)) {
            dead = true;
            atomicOr(a.status, 2);
        }
    };

    const int t = tid & (kFtRowThreads - 1);      // TMEM lane t
    const int g = gbase + t;                      // this CTA's physical row in lane t
    const bool valid = t < nr;
    const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const float2 kzv = a.kz2[kz];
    int cur = 0;

    if (warp >= kFtRowWarps) {
        // ------------------------------------------------------- helpers
        const bool issuer = warp == kFtRowWarps;   // its lane 0 issues the MMAs
        const uint32_t bhi = smem_u32(sm.Bhi), blo = smem_u32(sm.Blo);
        const uint32_t ybar_peer = mapa_u32(smem_u32(sm.y_bar), peer);
        const uint32_t yfree_peer = mapa_u32(smem_u32(sm.y_free), peer);
        const uint32_t y_peer = mapa_u32(smem_u32(sm.Y), peer);
        auto issue = [&](int c0, int len) { ft_issue(tmem, tmem + kXhi, tmem + kXlo, bhi, blo, c0, len); };
        uint32_t ph_x = 0, ph_bn = 0, ph_y = 0, ph_free = 0, ph_rest = 0;
        bool first = true;   // no panel before this one: Y is free
        if (lines > 0) ft_first_block<MID>(a, trow, valid, g, kz, MID ? hc.mid : hc.line(0), ncol, 1, kzv);
        tc_fence_before();
        ft_all_barrier();    // the first block is in TMEM
        tc_fence_after();
        for (int ls = 0; ls < lines; ls++) {
            for (int p = 0; p < npan; p++) {
                const int k0 = p * kFtB, bl = min(kFtB, n - k0);
                const bool next = p + 1 < npan;
                // the panel's steps are done and its X is in TMEM (the row
                // warps have waited for the previous trailing GEMM)
                wait_warp(sm.x_ready, ph_x);
                ph_x ^= 1u;
                if (issuer && next) {
                    wait_warp(sm.bn_ready, ph_bn);
                    ph_bn ^= 1u;
                    tc_fence_after();
                    if (lane == 0) {
                        issue(2 * kFtB * (p + 1), 2 * kFtB);
                        umma_commit(sm.next_ready);
                    }
                    __syncwarp();
                }
                tc_fence_after();
                if (!first) {   // the peer has read the previous panel's Y
                    wait_cluster(sm.y_free, ph_free);
                    ph_free ^= 1u;
                }
                first = false;
                // ---- this CTA's pivot rows (before the panel's update) in the
                // columns outside panels p and p + 1 into Y of both CTAs, two
                // 32-column loads in flight per wait
                const int skip = next ? 2 : 1, nc = npan - skip;
                const int my_step = valid ? sm.stepof[g] : -1;
                const bool piv = valid && my_step >= k0 && my_step < k0 + bl;
                if (__any_sync(0xffffffffu, piv)) {
                    const int yr = piv ? my_step - k0 : 0;
                    float2 *yrow = sm.Y + (size_t)yr * kF2Yld;
                    const uint32_t yrp = y_peer + (uint32_t)(yr * kF2Yld * sizeof(float2));
#pragma unroll 1
                    for (int c = 0; c < nc; c += 2) {
                        const int c0 = c < p ? c : c + skip, c1 = c + 1 < p ? c + 1 : c + 1 + skip;
                        float f[2][32];
                        tmem_ld32_nowait(trow + (uint32_t)(32 * c0), f[0]);
                        if (c + 1 < nc) tmem_ld32_nowait(trow + (uint32_t)(32 * c1), f[1]);
                        tmem_wait_ld(f[0]);
                        tmem_wait_ld(f[1]);
                        if (piv) {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                if (c + h >= nc) break;
                                const int col = 16 * (h ? c1 : c0);
#pragma unroll
                                for (int e = 0; e < 8; e++) {
                                    const float4 q4 = make_float4(f[h][4 * e], f[h][4 * e + 1], f[h][4 * e + 2],
                                                                  f[h][4 * e + 3]);
                                    reinterpret_cast<float4 *>(yrow + col)[e] = q4;
                                    st_cluster_v4f32(yrp + (uint32_t)((col + 2 * e) * sizeof(float2)), q4);
                                }
                            }
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive_warp_cluster(ybar_peer);
                ft_helper_barrier();
                wait_cluster(sm.y_bar, ph_y);
                ph_y ^= 1u;
                // ---- their B, and the GEMM of every column outside panels p, p + 1
                for (int c = 0; c < nc; c++) {
                    const int v = 128 * (c < p ? c : c + skip) + t;
                    const int kk0 = 2 * ((v >> 2) & 7), j = (v >> 5) * 4 + (v & 3);
                    const float2 y0 = kk0 < bl ? sm.Y[(size_t)kk0 * kF2Yld + j] : make_float2(0.f, 0.f);
                    const float2 y1 = kk0 + 1 < bl ? sm.Y[(size_t)(kk0 + 1) * kF2Yld + j] : make_float2(0.f, 0.f);
                    ft_put_b(sm.Bhi, sm.Blo, v, y0, y1);
                }
                fence_proxy_async_smem();
                mbar_arrive_warp_cluster(yfree_peer);
                ft_helper_barrier();
                tc_fence_after();
                if (issuer && lane == 0) {
                    issue(0, 2 * kFtB * p);
                    if (next) issue(2 * kFtB * (p + 2), 2 * ncol - 2 * kFtB * (p + 2));
                    umma_commit(sm.rest_done);
                }
                __syncwarp();
                if (next) ph_rest ^= 1u;   // (waited for by the row warps)
            }
            wait_warp(sm.rest_done, ph_rest);
            ph_rest ^= 1u;
            tc_fence_after();
            ft_all_barrier();   // the next frame
            cur ^= 1;
            {
                const int i = valid ? sm.rho[cur * kF2Tab + g] : 0;
                const bool more = ls + 1 < lines;
                const int line = MID ? hc.mid : hc.line(ls), nl = more ? hc.line(ls + 1) : 0;
                ft_line_out(a, trow, valid, i, sm.kap + cur * kF2Tab, sm.kapinv,
                            a.Gt + ((long)kz * a.ny + line) * (long)n * a.ldg, ncol, 1, more, nl,
                            more ? cmul(cin[nl], cout[line]) : make_float2(0.f, 0.f), kzv);
            }
            tc_fence_before();
            ft_all_barrier();   // the next line's block is in TMEM
            tc_fence_after();
        }
        if (issuer && lane == 0) {
            umma_commit(sm.fin);
            mbar_wait_bounded_cta(smem_u32(sm.fin), 0u, kFtWaitLimit);
        }
        __syncwarp();
    } else {
        // ----------------------------------------------------- row threads
        const int g1 = t + kFtRowThreads;        // the second row of the panel steps (g0 = t)
        const bool has1 = g1 < n;
        const uint32_t panbar_peer = mapa_u32(smem_u32(sm.pan_bar), peer);
        const uint32_t ynbar_peer = mapa_u32(smem_u32(sm.yn_bar), peer);
        const uint32_t pf_peer = mapa_u32(smem_u32(sm.PF), peer);
        const uint32_t yn_peer = mapa_u32(smem_u32(sm.Yn), peer);
        uint32_t ph_pan = 0, ph_yn = 0, ph_next = 0, ph_rest = 0;

        if (lines > 0) ft_first_block<MID>(a, trow, valid, g, kz, MID ? hc.mid : hc.line(0), ncol, 0, kzv);
        tc_fence_before();
        ft_all_barrier();
        tc_fence_after();

        for (int ls = 0; ls < lines; ls++) {
            const int line = MID ? hc.mid : hc.line(ls);
            bool used0 = false, used1 = false;
            for (int p = 0; p < npan; p++) {
                const int k0 = p * kFtB, bl = min(kFtB, n - k0);
                if (p > 0) {
                    wait_warp(sm.next_ready, ph_next);
                    ph_next ^= 1u;
                }
                // ---- this CTA's rows of the panel into both CTAs' PF
                {
                    float f[32];
                    tc_fence_after();
                    tmem_ld32_nowait(trow + (uint32_t)(2 * k0), f);
                    tmem_wait_ld(f);
                    if (valid) {
                        float4 *dst = reinterpret_cast<float4 *>(sm.PF + (size_t)g * kF2PFld);
                        const uint32_t rdst = pf_peer + (uint32_t)(g * kF2PFld * sizeof(float2));
#pragma unroll
                        for (int e = 0; e < kFtB / 2; e++) {
                            const float4 q4 = make_float4(f[4 * e], f[4 * e + 1], f[4 * e + 2], f[4 * e + 3]);
                            dst[e] = q4;
                            st_cluster_v4f32(rdst + 16u * (uint32_t)e, q4);
                        }
                    }
                    mbar_arrive_warp_cluster(panbar_peer);
                }
                ft_row_barrier();
                wait_cluster(sm.pan_bar, ph_pan);
                ph_pan ^= 1u;
                float2 P0[kFtB], P1[kFtB];
                {
                    const float4 *s0 = reinterpret_cast<const float4 *>(sm.PF + (size_t)t * kF2PFld);
                    const float4 *s1 = reinterpret_cast<const float4 *>(sm.PF + (size_t)(has1 ? g1 : t) * kF2PFld);
#pragma unroll
                    for (int e = 0; e < kFtB / 2; e++) {
                        const float4 x0 = s0[e], x1 = s1[e];
                        P0[2 * e] = make_float2(x0.x, x0.y);
                        P0[2 * e + 1] = make_float2(x0.z, x0.w);
                        P1[2 * e] = make_float2(x1.x, x1.y);
                        P1[2 * e + 1] = make_float2(x1.z, x1.w);
                    }
                }
                // ---- the panel's pivot steps, in each CTA on the whole panel.
                // The rows rotate by one column per step, so that the column
                // of step kk is always P[0] (no register indexed by kk): after
                // step kk, P[e] holds panel column (kk + 1 + e) mod 16.
                // A pivot row is left unscaled in its step (its multiplier is
                // 0, its new column 1) and scaled by its 1 / pv after the
                // panel: every later step is linear in the row, so this gives
                // the same rows as scaling it in its step. Each step issues
                // the next step's warp reduction right after the update of
                // the next pivot column, before the other columns.
                float2 sc0 = make_float2(1.f, 0.f), sc1 = sc0;
                bool piv0 = false, piv1 = false, bad = false;
                uint32_t key0 = ft_key(P0[0], !used0, t);
                uint32_t key1 = ft_key(P1[0], has1 && !used1, g1);
                uint32_t key = key0 > key1 ? key0 : key1;
                uint32_t kw = __reduce_max_sync(0xffffffffu, key);
                // every row's 1 / candidate, under the reduction's latency: the
                // winner's goes out with its row, so that no reciprocal stands
                // between the barrier and the next pivot column
                float2 inv0 = pivot_inv0(P0[0]), inv1 = pivot_inv0(P1[0]);
#pragma unroll 1
                for (int kk = 0; kk < bl; kk++) {
                    const int k = k0 + kk, buf = k & 1;
                    st_shared_u32_if(lane == 0, smem_u32(&sm.wkey[buf * kFtRowWarps + warp]), kw);
                    {
                        // the winning row in register order, w[1 + e] = prow[e], with
                        // 1 / pivot in the pivot's place
                        const bool win = kw != 0u && key == kw, first = key0 == kw;
                        const uint32_t w = smem_u32(sm.wrow + (size_t)(buf * kFtRowWarps + warp) * kFtB);
                        const float2 h0 = make_float2(first ? inv0.x : inv1.x, first ? inv0.y : inv1.y);
#pragma unroll
                        for (int e = 0; e < kFtB / 2; e++)
                            st_shared_v4_if(win, w + 16u * (uint32_t)e,
                                            make_float4(e == 0 ? h0.x : first ? P0[2 * e].x : P1[2 * e].x,
                                                        e == 0 ? h0.y : first ? P0[2 * e].y : P1[2 * e].y,
                                                        first ? P0[2 * e + 1].x : P1[2 * e + 1].x,
                                                        first ? P0[2 * e + 1].y : P1[2 * e + 1].y));
                    }
                    ft_row_barrier();
                    const uint4 kv = *reinterpret_cast<const uint4 *>(sm.wkey + buf * kFtRowWarps);
                    const uint32_t kmax = max(max(kv.x, kv.y), max(kv.z, kv.w));
                    const int r = kmax != 0u ? 255 - (int)(kmax & 0xFFu) : -1;
                    const int wsel = (r & (kFtRowThreads - 1)) >> 5;   // the warp that holds row r
                    // the pivot row, rotated like the rows: prow[e] = column (kk + 1 + e) mod 16
                    const float4 *w = reinterpret_cast<const float4 *>(sm.wrow + (size_t)(buf * kFtRowWarps + wsel) * kFtB);
                    float2 prow[kFtB], pinv = make_float2(0.f, 0.f);
#pragma unroll
                    for (int e = 0; e < kFtB / 2; e++) {
                        const float4 q4 = w[e];
                        if (e == 0) pinv = make_float2(r < 0 ? 0.f : q4.x, r < 0 ? 0.f : q4.y);
                        else prow[2 * e - 1] = make_float2(q4.x, q4.y);
                        prow[2 * e] = make_float2(q4.z, q4.w);
                    }
                    // no finite candidate, or an exactly zero pivot: flagged (after
                    // the panel), the block is invalid
                    bad |= pinv.x == 0.f && pinv.y == 0.f;
                    st_shared_u32_if(t == 0, smem_u32(&sm.perm[k]), (uint32_t)(r >= 0 ? r : 0));
                    // row -= (c / pv) * pivot row, column k becomes -c / pv
                    const bool ip0 = t == r, ip1 = g1 == r;
                    float2 s0 = cmul(P0[0], pinv), s1 = cmul(P1[0], pinv);
                    s0 = make_float2(ip0 ? 0.f : s0.x, ip0 ? 0.f : s0.y);
                    s1 = make_float2(ip1 ? 0.f : s1.x, ip1 ? 0.f : s1.y);
                    sc0 = make_float2(ip0 ? pinv.x : sc0.x, ip0 ? pinv.y : sc0.y);
                    sc1 = make_float2(ip1 ? pinv.x : sc1.x, ip1 ? pinv.y : sc1.y);
                    used0 |= ip0;
                    used1 |= ip1;
                    piv0 |= ip0;
                    piv1 |= ip1;
                    st_shared_u32_if(ip0 || ip1, smem_u32(&sm.stepof[r >= 0 ? r : 0]), (uint32_t)k);
                    P0[0] = cfms(s0, prow[0], P0[1]);
                    P1[0] = cfms(s1, prow[0], P1[1]);
                    key0 = ft_key(P0[0], !used0, t);
                    key1 = ft_key(P1[0], has1 && !used1, g1);
                    key = key0 > key1 ? key0 : key1;
                    kw = __reduce_max_sync(0xffffffffu, key);
                    inv0 = pivot_inv0(P0[0]);
                    inv1 = pivot_inv0(P1[0]);
#pragma unroll
                    for (int e = 1; e < kFtB - 1; e++) {
                        P0[e] = cfms(s0, prow[e], P0[e + 1]);
                        P1[e] = cfms(s1, prow[e], P1[e + 1]);
                    }
                    P0[kFtB - 1] = ip0 ? make_float2(1.f, 0.f) : make_float2(-s0.x, -s0.y);
                    P1[kFtB - 1] = ip1 ? make_float2(1.f, 0.f) : make_float2(-s1.x, -s1.y);
                }
                if (bad && t == 0 && rank == 0) atomicOr(a.status, 1);
                // the panel's pivot rows scaled by their 1 / pv
                if (piv0) {
#pragma unroll
                    for (int e = 0; e < kFtB; e++) P0[e] = cmul(P0[e], sc0);
                }
                if (piv1) {
#pragma unroll
                    for (int e = 0; e < kFtB; e++) P1[e] = cmul(P1[e], sc1);
                }
                // ---- the panel after its steps back into PF, in column order
                // (P[e] holds column (bl + e) mod 16)
                {
                    float2 *d0 = sm.PF + (size_t)t * kF2PFld;
                    float2 *d1 = sm.PF + (size_t)(has1 ? g1 : t) * kF2PFld;
#pragma unroll
                    for (int e = 0; e < kFtB; e++) d0[(bl + e) & (kFtB - 1)] = P0[e];
                    if (has1) {
#pragma unroll
                        for (int e = 0; e < kFtB; e++) d1[(bl + e) & (kFtB - 1)] = P1[e];
                    }
                }
                ft_row_barrier();

                // ---- the previous panel's trailing GEMM is done: X and the
                // panel's own columns of this CTA's rows into TMEM
                if (p > 0) {
                    wait_warp(sm.rest_done, ph_rest);
                    ph_rest ^= 1u;
                }
                tc_fence_after();
                const int my_step = valid ? sm.stepof[g] : -1;
                const bool piv = valid && my_step >= k0 && my_step < k0 + bl;
                {
                    float xh[32], xl[32], f[32];
                    const float4 *src = reinterpret_cast<const float4 *>(sm.PF + (size_t)(valid ? g : 0) * kF2PFld);
#pragma unroll
                    for (int e = 0; e < kFtB / 2; e++) {
                        const float4 q4 = src[e];
                        f[4 * e] = q4.x;
                        f[4 * e + 1] = q4.y;
                        f[4 * e + 2] = q4.z;
                        f[4 * e + 3] = q4.w;
                    }
                    if (!valid) {
#pragma unroll
                        for (int e = 0; e < 32; e++) f[e] = 0.f;
                    }
#pragma unroll
                    for (int e = 0; e < kFtB; e++) {
                        float2 x = make_float2(0.f, 0.f);
                        if (e < bl) {
                            x = make_float2(f[2 * e], f[2 * e + 1]);
                            if (piv && my_step == k0 + e) x.x -= 1.f;
                        }
                        tf32_split_fast(x.x, xh[2 * e], xl[2 * e]);
                        tf32_split_fast(x.y, xh[2 * e + 1], xl[2 * e + 1]);
                    }
                    tmem_st32(trow + kXhi, xh);
                    tmem_st32(trow + kXlo, xl);
                    tmem_st32(trow + (uint32_t)(2 * k0), f);
                    tmem_wait_st();
                }
                tc_fence_before();
                mbar_arrive_warp(sm.x_ready);
                if (p + 1 == npan) continue;   // no next panel
                // every read of this panel's PF is done before this CTA's
                // pivot rows go out (the peer writes the next panel's PF only
                // after it has them)
                ft_row_barrier();
                // ---- the panel's pivot rows of this CTA (their values before
                // the panel's update) in the next panel's columns into Yn of
                // both CTAs
                if (__any_sync(0xffffffffu, piv)) {
                    const int yr = piv ? my_step - k0 : 0;
                    float4 *yrow = reinterpret_cast<float4 *>(sm.Yn + (size_t)yr * kF2PFld);
                    const uint32_t yrp = yn_peer + (uint32_t)(yr * kF2PFld * sizeof(float2));
                    float f[32];
                    tmem_ld32_nowait(trow + (uint32_t)(32 * (p + 1)), f);
                    tmem_wait_ld(f);
                    if (piv) {
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const float4 q4 = make_float4(f[4 * e], f[4 * e + 1], f[4 * e + 2], f[4 * e + 3]);
                            yrow[e] = q4;
                            st_cluster_v4f32(yrp + 16u * (uint32_t)e, q4);
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive_warp_cluster(ynbar_peer);
                ft_row_barrier();
                wait_cluster(sm.yn_bar, ph_yn);
                ph_yn ^= 1u;
                // ---- their B: one unit per thread
                {
                    const int kk0 = 2 * ((t >> 2) & 7), j = (t >> 5) * 4 + (t & 3);
                    const float2 *y = sm.Yn + (size_t)kk0 * kF2PFld + j;
                    ft_put_b(sm.Bhi, sm.Blo, 128 * (p + 1) + t, y[0], y[kF2PFld]);
                }
                fence_proxy_async_smem();
                mbar_arrive_warp(sm.bn_ready);
            }

            // ---- the line's last GEMM done: the next frame
            wait_warp(sm.rest_done, ph_rest);
            ph_rest ^= 1u;
            tc_fence_after();
            ft_row_barrier();
            const int nxt = cur ^ 1;
            const int *rho = sm.rho + cur * kF2Tab, *kap = sm.kap + cur * kF2Tab;
            int *rho2 = sm.rho + nxt * kF2Tab, *kap2 = sm.kap + nxt * kF2Tab;
            ft_next_frame(n, t, rho, kap, rho2, kap2, sm.kapinv, sm.perm, sm.stepof);
            cur = nxt;

            // ---- G_line^T to global in the new frame, and S_{line+1} in place,
            // every other chunk by the helpers
            ft_all_barrier();
            {
                const bool more = ls + 1 < lines;
                const int nl = more ? hc.line(ls + 1) : 0;
                ft_line_out(a, trow, valid, valid ? rho2[g] : 0, kap2, sm.kapinv,
                            a.Gt + ((long)kz * a.ny + line) * (long)n * a.ldg, ncol, 0, more, nl,
                            more ? cmul(cin[nl], cout[line]) : make_float2(0.f, 0.f), kzv);
            }
            tc_fence_before();
            ft_all_barrier();   // the next line's block is in TMEM
            tc_fence_after();
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer is done with this CTA's shared memory
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kF2Cols);
}

bool factor_tc2_supported(bool c64, int n) { return c64 && n > 128 && n <= kF2MaxN; }

int launch_factor_tc2(const FactorArgs &fa, cudaStream_t st) {
    if (fa.n <= 128 || fa.n > kF2MaxN) return HELM3D_ERR_ARG;
    if (kF2SmemBytes > device_info().smem_optin) return HELM3D_ERR_ARG;
    return launch_pairs(fa.middle ? factor_tc2_kernel<true> : factor_tc2_kernel<false>, (fa.middle ? 1 : 2) * fa.nz,
                        kFtThreads, kF2SmemBytes, ft_args(fa), st);
}

}  // namespace h3d
