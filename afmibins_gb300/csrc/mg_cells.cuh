// Multigrid transfer arithmetic of one coarse cell, shared by the level
// kernels (kernels_mg.cu) and the V-cycle tail (kernels_tail.cu) so that every
// form of a transfer gives the same bits.
//
// The weights are tensor products, (1,3,3,1)^3/512 and (3,1)^3/64, so both
// transfers are evaluated axis by axis with explicit fused multiply-adds and
// one scaling by a power of two: 63 additions and FMAs per coarse cell in a
// tree of depth 10 for the restriction instead of a chain of 64 dependent
// FMAs (about 40 clocks each in FP64), and 4 operations per fine cell instead
// of 9 for the prolongation; on the FP64 pipe both matter. Weights and
// scalings are exact, so the rounding is that of the sums alone.
#pragma once

#include "common.cuh"

namespace afmib {

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// f0 + 3 f1 + 3 f2 + f3
template <typename T>
__device__ __forceinline__ T full4(T f0, T f1, T f2, T f3) {
    return fma_t(T(3), f1 + f2, f0 + f3);
}
// 3 near + far
template <typename T>
__device__ __forceinline__ T near4(T near, T far) {
    return fma_t(T(3), near, far);
}

// the (1,3,3,1)^2-weighted sum of a plane's 16 taps get(ky, kx): x, then y
template <typename T, typename G>
__device__ __forceinline__ T restrict_plane(G get) {
    T r[4];
#pragma unroll
    for (int ky = 0; ky < 4; ++ky) r[ky] = full4<T>(get(ky, 0), get(ky, 1), get(ky, 2), get(ky, 3));
    return full4<T>(r[0], r[1], r[2], r[3]);
}
// src/mg/solver.h:153-181: taps get(kz, ky, kx)
template <typename T, typename G>
__device__ __forceinline__ T restrict_taps(G get) {
    T p[4];
#pragma unroll
    for (int kz = 0; kz < 4; ++kz) p[kz] = restrict_plane<T>([&](int ky, int kx) { return get(kz, ky, kx); });
    return full4<T>(p[0], p[1], p[2], p[3]) * T(1.0 / 512.0);
}

// src/mg/solver.h:71-151. One fine plane of a coarse cell and its +1
// neighbours: n** on the near coarse plane, f** on the far one, second letter
// b, u along y and third l, r along x. put(rx, ry, value, scale): the fine cell
// nearest to corner (rx, ry) takes scale * value.
template <typename T, typename P>
__device__ __forceinline__ void prolong_plane4(T nbl, T nbr, T nul, T nur, T fbl, T fbr, T ful, T fur, P put) {
    const T bl = near4(nbl, fbl), br = near4(nbr, fbr), ul = near4(nul, ful), ur = near4(nur, fur);  // z
    const T l0 = near4(bl, ul), r0 = near4(br, ur), l1 = near4(ul, bl), r1 = near4(ur, br);          // y
    const T s = T(1.0 / 64.0);
    put(0, 0, near4(l0, r0), s);
    put(1, 0, near4(r0, l0), s);
    put(0, 1, near4(l1, r1), s);
    put(1, 1, near4(r1, l1), s);
}
// The two fine cells of a channel wall row (no y neighbour), or of a row of a
// 2D grid (near and far coarse rows in y): near row n, far row f.
template <typename T, typename P>
__device__ __forceinline__ void prolong_row2(T nl, T nr, T fl, T fr, P put) {
    const T l = near4(nl, fl), r = near4(nr, fr);
    const T s = T(1.0 / 16.0);
    put(0, near4(l, r), s);
    put(1, near4(r, l), s);
}

}  // namespace afmib
