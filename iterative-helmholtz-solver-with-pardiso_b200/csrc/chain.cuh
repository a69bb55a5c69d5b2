// chain.cuh -- the two-ended order of a kz system's y-lines, shared by the
// factor and sweep kernels.
//
// The block tridiagonal system over the ny lines is eliminated from both ends
// towards the middle line mid = ny / 2: half 0 takes lines 0 .. mid - 1 in
// order, half 1 lines ny - 1 .. mid + 1, and the middle line, whose Schur
// complement has a term from each half, comes last.  The two halves are
// independent chains of half the length, so a kz system occupies two CTAs
// (or CTA pairs) for half as many dependent steps.  With h's couplings
//   cin[line]   towards the line before it in h's order (cmy for half 0, cpy
//               for half 1),
//   cout[line]  towards the line after it (cpy, cmy),
// the factor is S = D_line - cin[line] cout[prev] G_prev in each half, and
//   S_mid = D_mid - cmy[mid] cpy[mid-1] G_{mid-1} - cpy[mid] cmy[mid+1] G_{mid+1};
// the solve is
//   forward   y_line = G_line (f_line - cin[line] y_prev)
//   middle    x_mid = G_mid (f_mid - cmy[mid] y_{mid-1} - cpy[mid] y_{mid+1})
//   backward  x_line = y_line - cout[line] G_line x_next.
#pragma once

namespace h3d {

struct HalfChain {
    int half, ny, mid, K;   // K: lines of this half before the middle one
    __device__ __forceinline__ HalfChain(int ny_, int half_)
        : half(half_), ny(ny_), mid(ny_ >> 1), K(half_ ? ny_ - 1 - (ny_ >> 1) : (ny_ >> 1)) {}
    // the s-th line of the half (s = K: the middle line)
    __device__ __forceinline__ int line(int s) const { return half ? ny - 1 - s : s; }
    // the sweep's steps: K forward, the middle, K backward
    __device__ __forceinline__ int steps() const { return 2 * K + 1; }
    __device__ __forceinline__ int step_line(int t) const { return line(t <= K ? t : 2 * K - t); }
    // whether the other half has lines, and its last one (the middle's neighbour)
    __device__ __forceinline__ bool peer_lines() const { return half ? mid > 0 : ny - 1 - mid > 0; }
    __device__ __forceinline__ int peer_last() const { return half ? mid - 1 : mid + 1; }
};

}  // namespace h3d
