// sweep.cu -- block sweep over y-lines for every kz (the per-kz 2D solve;
// replaces PARDISO phase 33, Source/functions.cpp:5959, and
// DirSolveFastDiagStruct, Source/HODLR/BinaryTreesHODLR.cpp:2971-3018).
//
// With G_j = S_j^{-1} from the factor, eliminated from both ends (chain.cuh):
// a cluster of two CTAs per kz, CTA h taking half h's lines: forward to the
// middle line, which both CTAs solve (from the other's last y, read from the
// planes), and back, in place on the plane of the kz.  A chain of ny lines is
// bound by the latency of its dependent lines, and the halves run side by side.
//
// G_j^T (row m = column m of G, contiguous) streams from HBM through a ring
// of shared-memory stages filled by 1D bulk copies (cp.async.bulk with
// mbarrier completion) that a dedicated producer warp issues as far ahead as
// the ring allows, independently of the line-to-line dependence chain.
// Each of the CW consumer warps owns RW = 32/G rows of y: lane (il, g) owns
// row i = w*RW + il and accumulates G^T[m][i] v[m][r] over the rows m = g,
// g+G, ... of every stage for all RR right-hand sides r (one G element feeds
// RR complex FMAs); the G partial sums of a row meet by warp shuffles.  The
// row owner also forms the next line's v[i][r] into a double-buffered shared
// array, so a y-line ends with one named barrier among the consumer warps and
// no shared-memory reduction.  What a line needs besides G v (the next line's
// right-hand side, or this line's y) is prefetched into registers while the
// line streams.  Planes of R right-hand sides are laid out [kz][line][r][i].
#include <cuda_runtime.h>

#include <cstdlib>

#include <cstdint>

#include "chain.cuh"
#include "cplx.cuh"
#include "helm3d_internal.h"
#include "ptx.cuh"

namespace h3d {

template <typename R> struct SweepK {
    int n, ny, ldg, nrhs;
    int groups, gsize;   // the right-hand sides in groups of gsize, a cluster of its own for each (kz, group)
    const cplx<R> *Gt;
    const cplx<R> *cmy, *cpy;
    cplx<R> *planes;
    const cplx<R> *dxy;  // adjoint: [2][ny][n] = alpha_x alpha_y, conj(1 / (alpha_x alpha_y))
    int rows_per_stage;  // rows of G^T per ring stage
    int nstage;          // ring depth
    uint32_t stage_bytes;
    int *status;
    uint32_t wait_limit;  // polls of a producer/consumer wait before it gives up (status bit 2)
    int expire_test;      // HELM3D_TEST_EXPIRE_WAIT: the consumers first wait on a barrier that
                          // nothing arrives on, so that the wait expires (tests of the status path)
    const int *kzslot;    // >= 0: a skipped mode (launch_kzskip_apply handles it), or null
};

// Polls of a bounded wait.  Waits between the producer and the consumers use
// SweepK::wait_limit (this value unless HELM3D_WAIT_LIMIT sets it, to make
// a wait expire in a test); the final drain of the producer's own copies
// always uses this value, so that no copy is in flight when the CTA exits.
constexpr uint32_t kSweepWaitLimit = 1u << 20;
constexpr int kSweepMaxN = 256;

template <int CW> __device__ __forceinline__ void consumer_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");
}

// The producer lane: streams the stages (rows_per_stage rows of G^T, cpl to a
// line) of every step of the half's chain into the ring, then waits (bounded)
// for its last copies to land, so that no bulk copy into this CTA's shared
// memory is still in flight when the CTA can exit.
template <typename R>
__device__ __forceinline__ void sweep_produce(const SweepK<R> &a, const HalfChain &hc, int kz, cplx<R> *ring,
                                              uint64_t *full, uint64_t *empty, int cpl) {
    const uint32_t row_bytes = (uint32_t)a.ldg * (uint32_t)sizeof(cplx<R>);
    RingPos rp;
    long issued = 0;
    bool stop = false;
    for (int t = 0; t < hc.steps() && !stop; t++) {
        const cplx<R> *src = a.Gt + ((long)kz * a.ny + hc.step_line(t)) * a.n * (long)a.ldg;
        for (int ch = 0; ch < cpl; ch++) {
            if (issued >= a.nstage && !mbar_wait_bounded_cta(smem_u32(&empty[rp.slot]), rp.phase ^ 1u, a.wait_limit)) {
                // stop issuing: the consumers' bounded waits on full[] expire in turn
                atomicOr(a.status, 4);
                stop = true;
                break;
            }
            const int r0 = ch * a.rows_per_stage;
            const uint32_t bytes = (uint32_t)min(a.rows_per_stage, a.n - r0) * row_bytes;
            mbar_expect_tx(&full[rp.slot], bytes);
            bulk_g2s(ring + (size_t)rp.slot * (a.stage_bytes / sizeof(cplx<R>)), src + (long)r0 * a.ldg, bytes,
                     &full[rp.slot]);
            rp.next(a.nstage);
            issued++;
        }
    }
    // the last use of every slot (rp is one past the final use)
    for (int k = 0; k < a.nstage && k < issued; k++) {
        int sl = rp.slot - 1 - k;
        uint32_t ph = rp.phase;
        if (sl < 0) {
            sl += a.nstage;
            ph ^= 1u;
        }
        mbar_wait_bounded_cta(smem_u32(&full[sl]), ph, kSweepWaitLimit);
    }
}

// The meeting of the halves at the middle line.  Each consumer warp has
// stored its rows' last forward y to the planes and arrives (release, cluster
// scope) on the peer's `met`; once its own `met` is complete the peer's y may
// be read from the planes.  Having read it, the warp arrives on the peer's
// `read`, which the peer waits for before its first backward step overwrites
// that line.
__device__ __forceinline__ void sweep_arrive_peer(uint64_t *bar, uint32_t peer) {
    mbar_arrive_warp_cluster(mapa_u32(smem_u32(bar), peer));
}

// RS consecutive values of a row of v, by 16-byte loads
template <int RS> __device__ __forceinline__ void load_v(double2 (&w)[RS], const double2 *p) {
#pragma unroll
    for (int r = 0; r < RS; r++) w[r] = p[r];
}
template <int RS> __device__ __forceinline__ void load_v(float2 (&w)[RS], const float2 *p) {
    if constexpr (RS == 1) {
        w[0] = *p;
    } else {
#pragma unroll
        for (int r = 0; r < RS; r += 2) {
            const float4 q = *reinterpret_cast<const float4 *>(p + r);
            w[r] = make_float2(q.x, q.y);
            w[r + 1] = make_float2(q.z, q.w);
        }
    }
}

// G groups of lanes split the rows m of each stage; RR right-hand sides.
// ADJ: the conjugate-transposed solve S^{-H} v = conj(Dxy)^{-1} conj(S^{-1}
// (Dxy conj(v))), Dxy = diag(alpha_x(i) alpha_y(j)): Dxy^{-1} S is complex
// symmetric (every coupling is alpha(node) alpha(half node) / h^2), so the
// same factor serves; the input is scaled and conjugated where it is loaded
// and the output where it is stored.
template <typename R, bool ADJ>
__device__ __forceinline__ cplx<R> adj_in(const SweepK<R> &a, int line, int i, cplx<R> f) {
    if (!ADJ) return f;
    return cmul(a.dxy[(long)line * a.n + i], mkc<R>(f.x, -f.y));
}
template <typename R, bool ADJ>
__device__ __forceinline__ cplx<R> adj_out(const SweepK<R> &a, int line, int i, cplx<R> x) {
    if (!ADJ) return x;
    return cmul(mkc<R>(x.x, -x.y), a.dxy[(long)(a.ny + line) * a.n + i]);
}

template <typename R, int G, int RR, bool ADJ, int CW>
__global__ void __launch_bounds__((CW + 1) * 32, 1) sweep_kernel(SweepK<R> a) {
    typedef cplx<R> Cx;
    constexpr int RW = 32 / G;  // rows of y per warp
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int n = a.n, ldg = a.ldg, Rs = a.nrhs;
    const int kz = (blockIdx.x >> 1) / a.groups, rg = (blockIdx.x >> 1) % a.groups * a.gsize;
    const int Rn = min(a.gsize, Rs - rg);   // this cluster's right-hand sides, rg, rg + 1, ...
    if (a.kzslot && a.kzslot[kz] >= 0) return;   // a skipped mode (kz_skip_ratio), in both CTAs
    const uint32_t rank = blockIdx.x & 1u, peer = rank ^ 1u;   // the rank in the cluster of two
    const HalfChain hc(a.ny, (int)rank);
    const int lane = threadIdx.x & 31, warp = warp_index();
    Cx *ring = reinterpret_cast<Cx *>(smem_raw);
    Cx *vbuf = reinterpret_cast<Cx *>(smem_raw + (size_t)a.nstage * a.stage_bytes);  // [2][n][RR]
    uint64_t *full = reinterpret_cast<uint64_t *>(vbuf + 2 * (size_t)n * RR);
    uint64_t *empty = full + a.nstage;
    uint64_t *never = empty + a.nstage;         // no thread arrives on it
    uint64_t *met = never + 1, *read = never + 2;   // the peer's consumer warps arrive on them
    Cx *P = a.planes + ((long)kz * a.ny * Rs + rg) * n;  // line j, rhs rg + r, row i at ((j*Rs + r)*n + i)
    const int cpl = (n + a.rows_per_stage - 1) / a.rows_per_stage;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.nstage; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CW);
        }
        mbar_init(never, 1);
        mbar_init(met, CW);
        mbar_init(read, CW);
        fence_mbar_init_cluster();
    }
    __syncthreads();
    cluster_arrive();   // the peer's barriers exist before the first remote arrive (waited below)

    if (warp == CW) {
        cluster_wait();
        if (lane == 0) sweep_produce(a, hc, kz, ring, full, empty, cpl);
        __syncwarp();
    } else {
        const int il = lane % RW, g = lane / RW;
        const int i = warp * RW + il;
        const bool own = i < n, fin = own && g == 0;
        bool dead = false;
        if (a.expire_test && !mbar_wait_warp_cta(smem_u32(never), 0u, a.wait_limit)) {
            dead = true;
            if (lane == 0) atomicOr(a.status, 4);
        }
        const Cx *cin = hc.half ? a.cpy : a.cmy, *cout = hc.half ? a.cmy : a.cpy;
        const int steps = hc.steps();
        auto load_f = [&](int line, int r) { return adj_in<R, ADJ>(a, line, i, P[((long)line * Rs + r) * n + i]); };
        // the middle line's input from its right-hand side f, this half's y and the peer's
        auto meet = [&](Cx (&v)[RR], const Cx (&y)[RR], const Cx (&f)[RR]) {
            sweep_arrive_peer(met, peer);
            if (!dead && !mbar_wait_warp_cluster(smem_u32(met), 0u, a.wait_limit)) {
                dead = true;
                if (lane == 0) atomicOr(a.status, 4);
            }
            Cx o[RR];
#pragma unroll
            for (int r = 0; r < RR; r++) {
                o[r] = mkc<R>(0, 0);
                if (fin && r < Rn && hc.peer_lines()) o[r] = P[((long)hc.peer_last() * Rs + r) * n + i];
            }
            const Cx cm = a.cmy[hc.mid], cp = a.cpy[hc.mid];
#pragma unroll
            for (int r = 0; r < RR; r++)
                v[r] = hc.half ? cfms(cp, y[r], cfms(cm, o[r], f[r])) : cfms(cp, o[r], cfms(cm, y[r], f[r]));
            sweep_arrive_peer(read, peer);
        };
        cluster_wait();
        {   // the first line's input
            Cx v[RR];
#pragma unroll
            for (int r = 0; r < RR; r++) v[r] = fin && r < Rn ? load_f(hc.line(0), r) : mkc<R>(0, 0);
            if (hc.K == 0) {
                Cx y[RR], f[RR];
#pragma unroll
                for (int r = 0; r < RR; r++) {
                    y[r] = mkc<R>(0, 0);
                    f[r] = v[r];
                }
                meet(v, y, f);
            }
            if (fin)
#pragma unroll
                for (int r = 0; r < RR; r++) vbuf[(size_t)i * RR + r] = v[r];
        }
        consumer_barrier<CW>();
        RingPos rp;
        // this thread's element of the plane's line (r = 0), and the step
        // from one line to the next in the half's order
        Cx *Pl = P + (long)hc.line(0) * Rs * n + i;
        const long lstep = hc.half ? -(long)Rs * n : (long)Rs * n;
        const int cstep = hc.half ? -1 : 1;
        const Cx *cptr = cin + hc.line(0);   // forward: cin of the line; backward: cout
        for (int t = 0; t < steps; t++) {
            const bool fwd = t <= hc.K;
            if (t == hc.K + 1) cptr = cout + hc.line(hc.K);
            const Cx *v = vbuf + (t & 1) * n * RR;
            Cx *vnext = vbuf + ((t + 1) & 1) * n * RR;
            // prefetch: the next line's right-hand side (forward) or this line's y (backward)
            Cx pre[RR];
#pragma unroll
            for (int r = 0; r < RR; r++) {
                pre[r] = mkc<R>(0, 0);
                if (fin && r < Rn && t != hc.K) pre[r] = Pl[(t < hc.K ? lstep : 0) + r * n];
            }
            // the next line's cin (forward), this line's cout (backward)
            cptr += fwd ? cstep : -cstep;
            const Cx cc = t + 1 < hc.K || !fwd ? *cptr : mkc<R>(0, 0);
            // SPLIT: the products with Re G and Im G apart, half the dependent
            // FMAs per element (above 4 right-hand sides the registers do not
            // hold both, and their independent chains hide the latency)
            constexpr bool SPLIT = RR <= 4;
            Cx acc[RR], acd[SPLIT ? RR : 1];
#pragma unroll
            for (int r = 0; r < RR; r++) {
                acc[r] = mkc<R>(0, 0);
                if constexpr (SPLIT) acd[r] = mkc<R>(0, 0);
            }
            for (int ch = 0; ch < cpl; ch++) {
                if (!dead && !mbar_wait_warp_cta(smem_u32(&full[rp.slot]), rp.phase, a.wait_limit)) {
                    dead = true;
                    if (lane == 0) atomicOr(a.status, 4);
                }
                const int r0 = ch * a.rows_per_stage;
                const int rows = min(a.rows_per_stage, n - r0);
                if (own) {
                    const Cx *st = ring + (size_t)rp.slot * (a.stage_bytes / sizeof(Cx)) + g * ldg + i;
                    const Cx *vm = v + (r0 + g) * RR;
                    auto add = [&](Cx gv, const Cx *wp) {
                        Cx w[RR];
                        load_v<RR>(w, wp);
#pragma unroll
                        for (int r = 0; r < RR; r++) {
                            if constexpr (SPLIT) {
                                acc[r].x = fma(gv.x, w[r].x, acc[r].x);
                                acc[r].y = fma(gv.x, w[r].y, acc[r].y);
                                acd[r].x = fma(gv.y, w[r].y, acd[r].x);
                                acd[r].y = fma(gv.y, w[r].x, acd[r].y);
                            } else {
                                acc[r] = cfma(gv, w[r], acc[r]);
                            }
                        }
                    };
                    // UB rows at a time, then the rest: short lines are all
                    // rest, so its loads too go ahead of its FMAs
                    constexpr int UB = RR > 2 ? 2 : G == 8 ? 4 : 8;
                    int ml = g;
                    for (; ml + (UB - 1) * G < rows; ml += UB * G, st += UB * G * ldg, vm += UB * G * RR) {
#pragma unroll
                        for (int u = 0; u < UB; u++) add(st[u * G * ldg], vm + u * G * RR);
                    }
                    Cx gv[UB - 1];
#pragma unroll
                    for (int u = 0; u < UB - 1; u++) gv[u] = ml + u * G < rows ? st[u * G * ldg] : mkc<R>(0, 0);
#pragma unroll
                    for (int u = 0; u < UB - 1; u++)
                        if (ml + u * G < rows) add(gv[u], vm + u * G * RR);
                }
                mbar_arrive_warp(&empty[rp.slot]);
                rp.next(a.nstage);
            }
#pragma unroll
            for (int r = 0; r < RR; r++) {
                if constexpr (SPLIT) {
                    acc[r].x -= acd[r].x;
                    acc[r].y += acd[r].y;
                }
#pragma unroll
                for (int off = RW; off < 32; off <<= 1) {
                    acc[r].x += __shfl_xor_sync(0xffffffffu, acc[r].x, off);
                    acc[r].y += __shfl_xor_sync(0xffffffffu, acc[r].y, off);
                }
            }
            // the peer has read this half's last y before it is overwritten
            if (t == hc.K + 1 && !dead && !mbar_wait_warp_cluster(smem_u32(read), 0u, a.wait_limit)) {
                dead = true;
                if (lane == 0) atomicOr(a.status, 4);
            }
            if (ADJ && t < hc.K) {
#pragma unroll
                for (int r = 0; r < RR; r++)
                    if (fin) pre[r] = adj_in<R, ADJ>(a, hc.line(t + 1), i, pre[r]);
            }
            Cx vn[RR];
#pragma unroll
            for (int r = 0; r < RR; r++) {
                Cx out;
                if (fwd) {
                    out = acc[r];                          // y_line, or x_mid
                    vn[r] = t == hc.K ? out : cfms(cc, out, pre[r]);
                } else {
                    out = cfms(cc, acc[r], pre[r]);        // x_line = y_line - cout G x_next
                    vn[r] = out;
                }
                if (fin && r < Rn && (t != hc.K || hc.half == 0))
                    Pl[r * n] = t >= hc.K ? adj_out<R, ADJ>(a, hc.step_line(t), i, out) : out;
            }
            if (t == hc.K - 1) meet(vn, acc, pre);
            if (fin) {
#pragma unroll
                for (int r = 0; r < RR; r++) vnext[i * RR + r] = vn[r];
            }
            Pl += fwd && t < hc.K ? lstep : -lstep;
            consumer_barrier<CW>();
        }
        __syncwarp();
    }
    cluster_sync_all();   // no CTA leaves while the peer may arrive on its barriers
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ void unpack2(uint64_t p, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
// two FP32 fused multiply-adds in one instruction
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Complex64 batches of RR >= 4, bound by the FP32 pipe and shared memory: a
// thread owns two adjacent rows (one 16-byte load of G) for all RR right-hand
// sides, so that a load of v feeds two products (one row per thread reads 34
// cycles of shared memory per 64 warp FMAs; this reads at most 36 per 128), two
// right-hand sides at a time in one instruction (fma2).  Lane il + RL g owns
// rows 2 il, 2 il + 1 of the warp's and adds up the rows m = g, g + G, ... of
// G^T; the G partial sums of a row meet by halving, which leaves each group g
// the right-hand sides from g RR / G on to finish.  Everything else as in
// sweep_kernel.  Sixteen sources, one row per thread -> this kernel: 32^3 84 ->
// 50 us, 64^3 291 -> 197, 96^3 1425 -> 830, 128^3 2461 -> 2030, 200 x 128 x 60
// 3080 -> 2880; eight: 64^3 141 -> 122, 96^3 765 -> 567, 128^3 1409 -> 1120.
// elements between the rows of v: the G rows that a warp reads at once lie in
// banks of their own
constexpr int kBatchPad = 2;

template <int G, int RR, bool ADJ, int CW>
__global__ void __launch_bounds__((CW + 1) * 32, 1) sweep_batch_kernel(SweepK<float> a) {
    typedef float2 Cx;
    constexpr int RL = 32 / G;                       // lanes along the rows
    constexpr int VS = RR + kBatchPad;                       // row stride of v
    constexpr int FS = RR >= G ? RR / G : 1;         // right-hand sides a thread finishes
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int n = a.n, ldg = a.ldg, Rs = a.nrhs;
    const int kz = (blockIdx.x >> 1) / a.groups, rg = (blockIdx.x >> 1) % a.groups * a.gsize;
    const int Rn = min(a.gsize, Rs - rg);   // this cluster's right-hand sides, rg, rg + 1, ...
    if (a.kzslot && a.kzslot[kz] >= 0) return;   // a skipped mode (kz_skip_ratio), in both CTAs
    const uint32_t rank = blockIdx.x & 1u, peer = rank ^ 1u;   // the rank in the cluster of two
    const HalfChain hc(a.ny, (int)rank);
    const int lane = threadIdx.x & 31, warp = warp_index();
    Cx *ring = reinterpret_cast<Cx *>(smem_raw);
    Cx *vbuf = reinterpret_cast<Cx *>(smem_raw + (size_t)a.nstage * a.stage_bytes);  // [2][n][RR]
    uint64_t *full = reinterpret_cast<uint64_t *>(vbuf + 2 * (size_t)n * VS);
    uint64_t *empty = full + a.nstage;
    uint64_t *never = empty + a.nstage;         // no thread arrives on it
    uint64_t *met = never + 1, *read = never + 2;   // the peer's consumer warps arrive on them
    Cx *P = a.planes + ((long)kz * a.ny * Rs + rg) * n;  // line j, rhs rg + r, row i at ((j*Rs + r)*n + i)
    const int cpl = (n + a.rows_per_stage - 1) / a.rows_per_stage;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.nstage; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CW);
        }
        mbar_init(never, 1);
        mbar_init(met, CW);
        mbar_init(read, CW);
        fence_mbar_init_cluster();
    }
    __syncthreads();
    cluster_arrive();   // the peer's barriers exist before the first remote arrive (waited below)

    if (warp == CW) {
        cluster_wait();
        if (lane == 0) sweep_produce(a, hc, kz, ring, full, empty, cpl);
        __syncwarp();
    } else {
        const int il = lane % RL, g = lane / RL;
        const int i = (warp * RL + il) * 2;
        const bool own = i < n;                      // (row i + 1 may be past n: ldg covers its loads)
        const int r0s = g * RR / G;                  // the first right-hand side this thread finishes
        const bool owner = own && (RR >= G || g % (G / RR) == 0);
        bool dead = false;
        if (a.expire_test && !mbar_wait_warp_cta(smem_u32(never), 0u, a.wait_limit)) {
            dead = true;
            if (lane == 0) atomicOr(a.status, 4);
        }
        const Cx *cin = hc.half ? a.cpy : a.cmy, *cout = hc.half ? a.cmy : a.cpy;
        const int steps = hc.steps();
        // element q of this thread's tile: row i + (q & 1), right-hand side r0s + (q >> 1)
        auto in = [&](int q) { return owner && i + (q & 1) < n && r0s + (q >> 1) < Rn; };
        auto at = [&](int line, int q) -> Cx & { return P[((long)line * Rs + r0s + (q >> 1)) * n + i + (q & 1)]; };
        auto meet = [&](Cx (&v)[2 * FS], const Cx (&f)[2 * FS]) {   // v: this half's y on entry
            sweep_arrive_peer(met, peer);
            if (!dead && !mbar_wait_warp_cluster(smem_u32(met), 0u, a.wait_limit)) {
                dead = true;
                if (lane == 0) atomicOr(a.status, 4);
            }
            const Cx cm = a.cmy[hc.mid], cp = a.cpy[hc.mid];
#pragma unroll
            for (int q = 0; q < 2 * FS; q++) {
                const Cx o = in(q) && hc.peer_lines() ? at(hc.peer_last(), q) : make_float2(0, 0);
                v[q] = hc.half ? cfms(cp, v[q], cfms(cm, o, f[q])) : cfms(cp, o, cfms(cm, v[q], f[q]));
            }
            sweep_arrive_peer(read, peer);
        };
        // v of a row: (x, x, y, y) of each pair of right-hand sides
        auto put = [&](Cx *vb, const Cx (&v)[2 * FS]) {
            if (!owner) return;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (i + h >= n) continue;
                float *row = reinterpret_cast<float *>(vb + (i + h) * VS);
                if constexpr (FS == 1) {
                    row[(r0s >> 1) * 4 + (r0s & 1)] = in(h) ? v[h].x : 0;
                    row[(r0s >> 1) * 4 + (r0s & 1) + 2] = in(h) ? v[h].y : 0;
                } else {
#pragma unroll
                    for (int f = 0; f < FS; f += 2) {
                        const Cx v0 = v[2 * f + h], v1 = v[2 * f + 2 + h];
                        const bool in0 = in(2 * f + h), in1 = in(2 * f + 2 + h);
                        reinterpret_cast<float4 *>(row)[(r0s + f) >> 1] =
                            make_float4(in0 ? v0.x : 0, in1 ? v1.x : 0, in0 ? v0.y : 0, in1 ? v1.y : 0);
                    }
                }
            }
        };
        cluster_wait();
        {   // the first line's input
            Cx v[2 * FS], f[2 * FS];
#pragma unroll
            for (int q = 0; q < 2 * FS; q++) {
                f[q] = in(q) ? adj_in<float, ADJ>(a, hc.line(0), i + (q & 1), at(hc.line(0), q)) : make_float2(0, 0);
                v[q] = make_float2(0, 0);
            }
            if (hc.K == 0) {
                meet(v, f);
                put(vbuf, v);
            } else {
                put(vbuf, f);
            }
        }
        consumer_barrier<CW>();
        RingPos rp;
        for (int t = 0; t < steps; t++) {
            const int line = hc.step_line(t);
            const bool fwd = t <= hc.K;
            const Cx *v = vbuf + (t & 1) * n * VS;
            Cx *vnext = vbuf + ((t + 1) & 1) * n * VS;
            // prefetch: the next line's right-hand side (forward) or this line's y (backward)
            Cx pre[2 * FS];
#pragma unroll
            for (int q = 0; q < 2 * FS; q++)
                pre[q] = in(q) && t != hc.K ? at(t < hc.K ? hc.line(t + 1) : line, q) : make_float2(0, 0);
            const Cx cc = t + 1 < hc.K ? cin[hc.line(t + 1)] : !fwd ? cout[line] : make_float2(0, 0);
            uint64_t ax[2][RR / 2], ay[2][RR / 2];   // real and imaginary parts of right-hand sides 2 r, 2 r + 1
#pragma unroll
            for (int r = 0; r < RR / 2; r++) ax[0][r] = ax[1][r] = ay[0][r] = ay[1][r] = 0;
            for (int ch = 0; ch < cpl; ch++) {
                if (!dead && !mbar_wait_warp_cta(smem_u32(&full[rp.slot]), rp.phase, a.wait_limit)) {
                    dead = true;
                    if (lane == 0) atomicOr(a.status, 4);
                }
                const int r0 = ch * a.rows_per_stage;
                const int rows = min(a.rows_per_stage, n - r0);
                if (own) {
                    const Cx *st = ring + (size_t)rp.slot * (a.stage_bytes / sizeof(Cx)) + g * ldg + i;
                    const Cx *vm = v + (r0 + g) * VS;
#pragma unroll 2
                    for (int ml = g; ml < rows; ml += G, st += G * ldg, vm += G * VS) {
                        const float4 gv = *reinterpret_cast<const float4 *>(st);
                        const uint64_t gx0 = pack2(gv.x, gv.x), gy0 = pack2(gv.y, gv.y), hy0 = pack2(-gv.y, -gv.y);
                        const uint64_t gx1 = pack2(gv.z, gv.z), gy1 = pack2(gv.w, gv.w), hy1 = pack2(-gv.w, -gv.w);
#pragma unroll
                        for (int r = 0; r < RR / 2; r++) {
                            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(vm + 2 * r);
                            ax[0][r] = fma2(hy0, w.y, fma2(gx0, w.x, ax[0][r]));
                            ay[0][r] = fma2(gy0, w.x, fma2(gx0, w.y, ay[0][r]));
                            ax[1][r] = fma2(hy1, w.y, fma2(gx1, w.x, ax[1][r]));
                            ay[1][r] = fma2(gy1, w.x, fma2(gx1, w.y, ay[1][r]));
                        }
                    }
                }
                mbar_arrive_warp(&empty[rp.slot]);
                rp.next(a.nstage);
            }
            Cx acc[2][RR];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int r = 0; r < RR / 2; r++) {
                    unpack2(ax[h][r], acc[h][2 * r].x, acc[h][2 * r + 1].x);
                    unpack2(ay[h][r], acc[h][2 * r].y, acc[h][2 * r + 1].y);
                }
            // the G partial sums: the group bit of each step keeps its half of
            // the right-hand sides (one left: plain sums)
#pragma unroll
            for (int s = G / 2, cnt = RR; s >= 1; s >>= 1) {
                const bool hi = (g & s) != 0;
                if (cnt > 1) {
                    cnt >>= 1;
#pragma unroll
                    for (int r = 0; r < RR / 2; r++)
                        if (r < cnt) {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const Cx lo = acc[h][r], up = acc[h][r + cnt];
                                const Cx send = hi ? lo : up;
                                Cx keep = hi ? up : lo;
                                keep.x += __shfl_xor_sync(0xffffffffu, send.x, RL * s);
                                keep.y += __shfl_xor_sync(0xffffffffu, send.y, RL * s);
                                acc[h][r] = keep;
                            }
                        }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        acc[h][0].x += __shfl_xor_sync(0xffffffffu, acc[h][0].x, RL * s);
                        acc[h][0].y += __shfl_xor_sync(0xffffffffu, acc[h][0].y, RL * s);
                    }
                }
            }
            // the peer has read this half's last y before it is overwritten
            if (t == hc.K + 1 && !dead && !mbar_wait_warp_cluster(smem_u32(read), 0u, a.wait_limit)) {
                dead = true;
                if (lane == 0) atomicOr(a.status, 4);
            }
            if (ADJ && t < hc.K) {
#pragma unroll
                for (int q = 0; q < 2 * FS; q++)
                    if (in(q)) pre[q] = adj_in<float, ADJ>(a, hc.line(t + 1), i + (q & 1), pre[q]);
            }
            Cx vn[2 * FS];
#pragma unroll
            for (int q = 0; q < 2 * FS; q++) {
                const Cx sum = acc[q & 1][q >> 1];
                const Cx out = fwd ? sum : cfms(cc, sum, pre[q]);   // y, x_mid, or x = y - cout G x_next
                vn[q] = t + 1 < hc.K ? cfms(cc, out, pre[q]) : out;
                if (in(q) && (t != hc.K || hc.half == 0))
                    at(line, q) = t >= hc.K ? adj_out<float, ADJ>(a, line, i + (q & 1), out) : out;
            }
            if (t == hc.K - 1) meet(vn, pre);
            put(vnext, vn);
            consumer_barrier<CW>();
        }
        __syncwarp();
    }
    cluster_sync_all();   // no CTA leaves while the peer may arrive on its barriers
}

// A launch of kern: CW consumer warps, rows of v of vs elements; even > 0: the
// stages of a line are the same multiple of that many rows; the right-hand
// sides in so many groups.
template <typename R, int CW>
static int sweep_go(void (*kern)(SweepK<R>), int vs, int even, int groups, const SweepArgs &sa, cudaStream_t st) {
    typedef cplx<R> Cx;
    SweepK<R> k;
    k.n = sa.n;
    k.ny = sa.ny;
    k.ldg = sa.ldg;
    k.nrhs = sa.R;
    k.groups = groups;
    k.gsize = (sa.R + groups - 1) / groups;
    k.Gt = (const Cx *)sa.Gt;
    k.cmy = (const Cx *)sa.cmy;
    k.cpy = (const Cx *)sa.cpy;
    k.planes = (Cx *)sa.planes;
    k.dxy = (const Cx *)sa.dxy;
    k.status = sa.status;
    k.kzslot = sa.kzslot;
    k.wait_limit = wait_limit_polls(kSweepWaitLimit);
    {
        const char *e = std::getenv("HELM3D_TEST_EXPIRE_WAIT");
        k.expire_test = (e && *e && *e != '0') ? 1 : 0;
    }
    const size_t vbytes = sizeof(Cx) * 2 * (size_t)sa.n * vs;
    const size_t budget = device_info().smem_optin - vbytes - 1024;
    // stages of about stage_kb (two at least fit), as many as fit the rest of
    // shared memory (at most ring_kb)
    const size_t row_bytes = (size_t)sa.ldg * sizeof(Cx);
    const size_t ring_max = (size_t)sa.ring_kb * 1024;
    const size_t ring_cap = budget < ring_max ? budget : ring_max;
    size_t stage = (size_t)sa.stage_kb * 1024;
    if (stage > ring_cap / 2 - 128) stage = ring_cap / 2 - 128;
    int rows = (int)(stage / row_bytes);
    if (rows < 1) rows = 1;
    if (even) {   // equal stages of a line, so that no group of lanes has more rows than another
        rows = rows < even ? even : rows / even * even;
        const int cpl = (sa.n + rows - 1) / rows, per = (sa.n + cpl - 1) / cpl;
        rows = (per + even - 1) / even * even;
    } else if (rows > sa.n) {
        rows = sa.n;
    }
    k.rows_per_stage = rows;
    k.stage_bytes = (uint32_t)(((size_t)rows * row_bytes + 127) & ~(size_t)127);
    int nst = (int)(ring_cap / k.stage_bytes);
    if (nst > 32) nst = 32;
    if (nst < 2) return HELM3D_ERR_ARG;
    k.nstage = nst;
    const size_t smem = (size_t)nst * k.stage_bytes + vbytes + (2 * nst + 3) * sizeof(uint64_t);
    return launch_pairs(kern, sa.nz * groups, (CW + 1) * 32, smem, k, st);
}

template <typename R, int G, int RR, bool ADJ, int CW> static int sweep_impl(const SweepArgs &sa, cudaStream_t st, int groups = 1) {
    return sweep_go<R, CW>(sweep_kernel<R, G, RR, ADJ, CW>, RR, 0, groups, sa, st);
}

// complex64 batches: 64 / G rows per warp.  More than 8 right-hand sides as two
// groups where that fills the last wave of CTAs (one to an SM above 64 rows): a
// group of 8 takes 0.55 of the time of 16 (96 x 96 x 64, one wave: 293 of 526
// us), so 96^3 x 16 as three waves of 8 instead of two of 16: 1032 ->
// 830 us (128^3, 4 waves of 8 for 2 of 16, stays).
template <int G, bool ADJ, int CW> static int sweep_batch(const SweepArgs &sa, cudaStream_t st) {
    if (sa.R <= 4) return sweep_go<float, CW>(sweep_batch_kernel<G, 4, ADJ, CW>, 4 + kBatchPad, G, 1, sa, st);
    if (sa.R <= 8) return sweep_go<float, CW>(sweep_batch_kernel<G, 8, ADJ, CW>, 8 + kBatchPad, G, 1, sa, st);
    const int sms = device_info().sm_count, one = (2 * sa.nz + sms - 1) / sms, two = (4 * sa.nz + sms - 1) / sms;
    if (sa.n > 64 && 11 * two < 20 * one)
        return sweep_go<float, CW>(sweep_batch_kernel<G, 8, ADJ, CW>, 8 + kBatchPad, G, 2, sa, st);
    return sweep_go<float, CW>(sweep_batch_kernel<G, 16, ADJ, CW>, 16 + kBatchPad, G, 1, sa, st);
}

// The split of a line over the consumer warps: 32 / G rows per warp, CW warps.
// One or two right-hand sides leave registers for 16 warps, which halves the
// elements each lane adds up in sequence; more take 8.
template <typename R, bool ADJ, int G1, int CW1, int G2> static int sweep_rr(const SweepArgs &sa, cudaStream_t s) {
    if (sa.R <= 1) return sweep_impl<R, G1, 1, ADJ, CW1>(sa, s);
    if (sa.R <= 2) return sweep_impl<R, G1, 2, ADJ, CW1>(sa, s);
    if constexpr (sizeof(R) == 8 || G2 == 4)
        if (sa.R <= 4) return sweep_impl<R, G2, 4, ADJ, 8>(sa, s);
    if constexpr (sizeof(R) == 8) {
        if (sa.R <= 8) return sweep_impl<R, G2, 8, ADJ, 8>(sa, s);
        // sums of 16 right-hand sides do not fit the registers (spilled, 64^3:
        // 957 us; two groups of 8, although they read G twice, 530)
        return sweep_impl<R, G2, 8, ADJ, 8>(sa, s, 2);
    }
    return HELM3D_ERR_ARG;   // (complex64 batches are sweep_batch's)
}

template <typename R, bool ADJ> static int sweep_n(const SweepArgs &sa, cudaStream_t s) {
    if constexpr (sizeof(R) == 4) {
        // (three or four sources of up to 64 rows: 88 us by sweep_kernel at 64^3,
        // 93 by this.)  Warps of 8 or 16 rows by whichever leaves the four
        // schedulers of an SM the same number: 16 sources of 96 rows are 1.2
        // times slower as 6 warps of 16 rows than as 12 of 8, of 160 rows 1.3
        // times as 5 of 32 than as 10 of 16, of 200 rows the same either way
        if (sa.R > 4 || (sa.R > 2 && sa.n > 64)) {
            if (sa.n <= 32) return sweep_batch<8, ADJ, 4>(sa, s);
            if (sa.n <= 64) return sweep_batch<8, ADJ, 8>(sa, s);
            if (sa.n <= 96) return sweep_batch<8, ADJ, 12>(sa, s);
            if (sa.n <= 128) return sweep_batch<4, ADJ, 8>(sa, s);
            if (sa.n <= 192) return sweep_batch<4, ADJ, 12>(sa, s);
            if (sa.n <= 240) return sweep_batch<4, ADJ, 15>(sa, s);
            return sweep_batch<2, ADJ, 8>(sa, s);
        }
    }
    if (sa.n <= 32) return sweep_rr<R, ADJ, 8, 8, 4>(sa, s);
    // complex64: 16 rows of a warp make 128 bytes, one shared-memory wavefront
    if (sa.n <= 64) return sweep_rr<R, ADJ, sizeof(R) == 4 ? 2 : 4, sizeof(R) == 4 ? 4 : 8, 4>(sa, s);
    if (sa.n <= 128) return sweep_rr<R, ADJ, 4, 16, 2>(sa, s);
    return sweep_rr<R, ADJ, 2, 16, 1>(sa, s);
}

void sweep_variant(int v, SweepArgs &a) {
    static const int kStage[kSweepVariants] = {32, 16, 64, 96, 32, 16, 0, 0, 0, 0};
    static const int kRingKb[kSweepVariants] = {200, 200, 200, 200, 100, 100, 0, 0, 0, 0};
    static const int kTcOcc[kSweepVariants] = {0, 0, 0, 0, 0, 0, 2, 2, 1, 1};
    static const int kTcStages[kSweepVariants] = {0, 0, 0, 0, 0, 0, 8, 4, 4, 8};
    if (v < 0 || v >= kSweepVariants) v = 0;
    a.stage_kb = kStage[v] ? kStage[v] : 32;
    a.ring_kb = kRingKb[v] ? kRingKb[v] : 200;
    a.tc_occ = kTcOcc[v];
    a.tc_stages = kTcStages[v];
}

bool sweep_variant_own(bool c64, int n, int v) { return v < 6 || (c64 && (n <= 128 || v < 8)); }

// The variant of a batch that no solve of this context has been tuned for:
// the CUDA-core kernel, whose products are FP32 (the tensor cores' FP16 hi/lo
// products add about a fifth to the complex64 preconditioner's error, 3.1e-6
// -> 3.8e-6 at 96^3, which a solve corrects and a caller's single apply does
// not).  A stage's first products wait for its first loads, so stages are
// large: complex64 by 96 KB where that holds a line or for several sources
// (96^3 against 64 KB: one source 312 -> 295 us, 16 sources 1074 -> 1032), by
// 64 KB for one or two of longer lines (128^3 with 96 KB 723 us, 64 KB 657)
// and for complex128 (one source, 128^3: 1286 us by 32 KB, 1248).  Below
// 32 KB a line is one stage either way.
int sweep_default(bool c64, int n, int R) {
    const size_t line = (size_t)n * n * (c64 ? 8 : 16);
    if (line <= 32 * 1024) return 0;
    return c64 && (R > 2 || line <= 96 * 1024) ? 3 : 2;
}

static int launch_sweep_kernels(bool c64, const SweepArgs &sa, cudaStream_t s);

int launch_sweep(bool c64, const SweepArgs &sa, cudaStream_t s) {
    const int rc = launch_sweep_kernels(c64, sa, s);
    if (rc || sa.nskip <= 0) return rc;
    return launch_kzskip_apply(c64, sa, s);   // the skipped modes, which the sweep kernels left
}

static int launch_sweep_kernels(bool c64, const SweepArgs &sa, cudaStream_t s) {
    if (sa.n < 1 || sa.n > kSweepMaxN || sa.R < 1 || sa.R > kMaxBatch) return HELM3D_ERR_ARG;
    // the tensor-core kernel where it applies (complex64, the packed factor, shared memory fits)
    if (c64 && sa.tc_occ && sweep_tcp_supported(sa)) return launch_sweep_tcp(sa, s);
    if (c64) return sa.dxy ? sweep_n<float, true>(sa, s) : sweep_n<float, false>(sa, s);
    return sa.dxy ? sweep_n<double, true>(sa, s) : sweep_n<double, false>(sa, s);
}

}  // namespace h3d
