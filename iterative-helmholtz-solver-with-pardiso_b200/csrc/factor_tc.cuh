// factor_tc.cuh -- parts shared by the tensor-core factors (factor_tc.cu, one
// CTA per block; factor_tc2.cu, a CTA pair): the block's entries, the pivot
// keys, the GEMM operand and the write-out of a finished line.
#pragma once
#include <cstdint>

#include "chain.cuh"
#include "cplx.cuh"
#include "helm3d_internal.h"
#include "ptx.cuh"
#include "tcgen05.cuh"

namespace h3d {

constexpr int kFtRowWarps = 4;
constexpr int kFtRowThreads = kFtRowWarps * 32;
constexpr int kFtThreads = 2 * kFtRowThreads;    // the row warps and as many helpers
constexpr int kFtB = 16;                         // panel width
constexpr uint32_t kFtWaitLimit = 1u << 22;

struct FtK {
    int n, ny, ldg;
    float2 *Gt;
    const float2 *cmx, *cpx, *cmy, *cpy, *base2d, *kz2;
    int *status;
    const int *kzslot;   // >= 0: a skipped mode (nothing to do), or null
};

inline FtK ft_args(const FactorArgs &fa) {
    FtK k;
    k.n = fa.n;
    k.ny = fa.ny;
    k.ldg = fa.ldg;
    k.Gt = (float2 *)fa.Gt;
    k.cmx = (const float2 *)fa.cmx;
    k.cpx = (const float2 *)fa.cpx;
    k.cmy = (const float2 *)fa.cmy;
    k.cpy = (const float2 *)fa.cpy;
    k.base2d = (const float2 *)fa.base2d;
    k.kz2 = (const float2 *)fa.kz2;
    k.status = fa.status;
    k.kzslot = fa.kzslot;
    return k;
}

__device__ __forceinline__ void ft_row_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(kFtRowThreads) : "memory");
}
__device__ __forceinline__ void ft_helper_barrier() {
    asm volatile("bar.sync 2, %0;" ::"n"(kFtThreads - kFtRowThreads) : "memory");
}
__device__ __forceinline__ void ft_all_barrier() { asm volatile("bar.sync 3, %0;" ::"n"(kFtThreads) : "memory"); }

// The tridiagonal D_line in logical row i: diagonal, and the couplings to
// logical columns i - 1 (sub) and i + 1 (sup).
struct FtDrow {
    float2 diag, sub, sup;
};
__device__ __forceinline__ FtDrow ft_drow(const FtK &a, int line, int i, float2 kzv) {
    FtDrow d;
    const float2 cyd = make_float2(-(a.cmy[line].x + a.cpy[line].x), -(a.cmy[line].y + a.cpy[line].y));
    d.diag = cadd(cadd(cyd, a.base2d[(long)line * a.n + i]), kzv);
    d.diag.x -= a.cmx[i].x + a.cpx[i].x;
    d.diag.y -= a.cmx[i].y + a.cpx[i].y;
    d.sub = a.cmx[i];
    d.sup = a.cpx[i];
    return d;
}

// pivot key of an entry of row g (0 when the row is not a candidate)
__device__ __forceinline__ uint32_t ft_key(float2 v, bool cand, int g) {
    if (!cand) return 0u;
    const float av = fabsf(v.x) + fabsf(v.y);
    if (!(av == av)) return 0u;
    return (__float_as_uint(av) & 0xFFFFFF00u) | (uint32_t)(255 - g);
}

// Unit v of the real form of Y (rows 2j + c, K = 2kk + c'), hi and lo, from the
// pivot rows' entries y0, y1 in column j = (v >> 5) * 4 + (v & 3), K quad
// kq = (v >> 2) & 7: the 16-byte units of rows 2j, (Re y, -Im y), and 2j + 1,
// (Im y, Re y), adjacent in address order (row & 7, K quad, 8-row group); the
// TF32 split is odd in its argument, so one split serves both rows.
__device__ __forceinline__ void ft_put_b(float *Bhi, float *Blo, int v, float2 y0, float2 y1) {
    float4 h, l;   // split of (Re y0, Im y0, Re y1, Im y1)
    tf32_split_fast(y0.x, h.x, l.x);
    tf32_split_fast(y0.y, h.y, l.y);
    tf32_split_fast(y1.x, h.z, l.z);
    tf32_split_fast(y1.y, h.w, l.w);
    const int u0 = (v >> 5) * 64 + ((v >> 2) & 7) * 8 + 2 * (v & 3);
    float4 *bh = reinterpret_cast<float4 *>(Bhi) + u0;
    float4 *bl = reinterpret_cast<float4 *>(Blo) + u0;
    bh[0] = make_float4(h.x, -h.y, h.z, -h.w);
    bh[1] = make_float4(h.y, h.x, h.w, h.z);
    bl[0] = make_float4(l.x, -l.y, l.z, -l.w);
    bl[1] = make_float4(l.y, l.x, l.w, l.z);
}

// G_line^T to global memory in the frame (kap, i = rho of the thread's row),
// and, with more, the next line's S in place: the 16-column chunks c = which,
// which + 2, ... of this thread's TMEM lane.
__device__ __forceinline__ void ft_line_out(const FtK &a, uint32_t trow, bool valid, int i, const int *kap,
                                            const int *kapinv, float2 *gout, int ncol, int which, bool more,
                                            int nl, float2 cc, float2 kzv) {
    const int n = a.n;
    FtDrow d = {};
    int qd = -1, qs = -1, qp = -1;
    if (more && valid) {
        d = ft_drow(a, nl, i, kzv);
        qd = kapinv[i];
        qs = i > 0 ? kapinv[i - 1] : -1;
        qp = i + 1 < n ? kapinv[i + 1] : -1;
    }
#pragma unroll 1
    for (int c = which; c < ncol / 16; c += 2) {
        float f[32];
        tmem_ld32_nowait(trow + (uint32_t)(32 * c), f);
        int kq[16];
#pragma unroll
        for (int e = 0; e < 4; e++) *reinterpret_cast<int4 *>(kq + 4 * e) = reinterpret_cast<const int4 *>(kap + 16 * c)[e];
        tmem_wait_ld(f);
#pragma unroll
        for (int e = 0; e < 16; e++) {   // (selects: a branch per entry costs more than the entry)
            const int q = 16 * c + e;
            const float2 m = make_float2(f[2 * e], f[2 * e + 1]);
            st_global_f2_if(valid && q < n, gout + (unsigned)(kq[e] * a.ldg + i), m);
            const float2 dd = make_float2(q == qd ? d.diag.x : q == qs ? d.sub.x : q == qp ? d.sup.x : 0.f,
                                          q == qd ? d.diag.y : q == qs ? d.sub.y : q == qp ? d.sup.y : 0.f);
            f[2 * e] = dd.x - (cc.x * m.x - cc.y * m.y);
            f[2 * e + 1] = dd.y - (cc.x * m.y + cc.y * m.x);
        }
        if (more) tmem_st32(trow + (uint32_t)(32 * c), f);
    }
    tmem_wait_st();
}

// The first line's block in the identity frame: D, and for the middle line
// (MID) both neighbours' terms, their G from global memory; the 16-column
// chunks which, which + 2, ... of row g.
template <bool MID>
__device__ __forceinline__ void ft_first_block(const FtK &a, uint32_t trow, bool valid, int g, int kz, int line,
                                               int ncol, int which, float2 kzv) {
    const int n = a.n;
    FtDrow d = {};
    if (valid) d = ft_drow(a, line, g, kzv);
    const bool lo = MID && line > 0, hi = MID && line + 1 < a.ny;
    const float2 clo = lo ? cmul(a.cmy[line], a.cpy[line - 1]) : make_float2(0.f, 0.f);
    const float2 chi = hi ? cmul(a.cpy[line], a.cmy[line + 1]) : make_float2(0.f, 0.f);
    const float2 *glo = a.Gt + ((long)kz * a.ny + line - 1) * (long)n * a.ldg + g;
    const float2 *ghi = glo + 2 * (long)n * a.ldg;
#pragma unroll 1
    for (int c = which; c < ncol / 16; c += 2) {
        float f[32];
#pragma unroll
        for (int e = 0; e < 16; e++) {
            const int q = 16 * c + e;
            const bool in = valid && q < n;
            float2 s = make_float2(!in ? 0.f : q == g ? d.diag.x : q == g - 1 ? d.sub.x : q == g + 1 ? d.sup.x : 0.f,
                                   !in ? 0.f : q == g ? d.diag.y : q == g - 1 ? d.sub.y : q == g + 1 ? d.sup.y : 0.f);
            if (MID) {
                if (lo && in) s = cfms(clo, glo[(long)q * a.ldg], s);
                if (hi && in) s = cfms(chi, ghi[(long)q * a.ldg], s);
            }
            f[2 * e] = s.x;
            f[2 * e + 1] = s.y;
        }
        tmem_st32(trow + (uint32_t)(32 * c), f);
    }
    tmem_wait_st();
}

// D[:, c0 + [0, len)) += X B[c0 + [0, len), :]^T, 3xTF32, in chunks of N <= 256
// (X in TMEM: hi at xhi, lo at xlo; B in shared memory: bhi, blo)
__device__ __forceinline__ void ft_issue(uint32_t tmem, uint32_t xhi, uint32_t xlo, uint32_t bhi, uint32_t blo, int c0,
                                         int len) {
    const uint32_t sbo = (uint32_t)(2 * kFtB / 4) * 128u;
    for (int off = 0; off < len; off += 256) {
        const int nn = len - off < 256 ? len - off : 256;
        const int col = c0 + off;
        const uint32_t idesc = umma_idesc_tf32(nn);
        const uint32_t boff = (uint32_t)(col / 8) * sbo;
#pragma unroll
        for (int ks = 0; ks < 2 * kFtB / 8; ks++) {
            const uint32_t koff = (uint32_t)ks * 256u;   // 8 K = two core matrices of 128 B
            const uint64_t dh = umma_desc(bhi + boff + koff, 128, sbo);
            const uint64_t dl = umma_desc(blo + boff + koff, 128, sbo);
            const uint32_t xh = xhi + (uint32_t)(ks * 8), xl = xlo + (uint32_t)(ks * 8);
            const uint32_t d = tmem + (uint32_t)col;
            umma_tf32_ts(d, xh, dh, idesc, 1u);
            umma_tf32_ts(d, xh, dl, idesc, 1u);
            umma_tf32_ts(d, xl, dh, idesc, 1u);
        }
    }
}

// The next frame from a finished line's pivots: rho' = kap o sigma, kap' = rho o
// perm, kapinv' (sigma = stepof, which is reset for the next line).  By the row
// warps; a barrier of all threads has to follow.
__device__ __forceinline__ void ft_next_frame(int n, int t, const int *rho, const int *kap, int *rho2, int *kap2,
                                              int *kapinv, const int *perm, int *stepof) {
    for (int q = t; q < n; q += kFtRowThreads) {
        int st = stepof[q];
        st = (st >= 0 && st < n) ? st : 0;   // a failed step leaves rows unpivoted (status set)
        rho2[q] = kap[st];
        kap2[q] = rho[perm[q]];
    }
    ft_row_barrier();
    for (int q = t; q < n; q += kFtRowThreads) {
        kapinv[kap2[q]] = q;
        stepof[q] = -1;
    }
}

}  // namespace h3d
