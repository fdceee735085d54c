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

constexpr int kOmegaMinNx = 64;  // smallest level (x extent) on which a requested over-relaxation applies

// A plain Gauss-Seidel sweep ends with the black colour, which leaves the
// residual zero on the black cells, so on levels without over-relaxation the
// residual is formed on the red cells only, the black ones count as zero in the
// restriction, and the prolongation leaves out the red cells, which the next
// sweep's red colour replaces without reading: half of each pass's work.
// FP64 levels, and FP32 ones below the over-relaxed sizes.
inline bool restrict_after_sweep(const Dims& d, size_t elem, int nu1) {
    return nu1 > 0 && (elem == sizeof(double) || d.nx < kOmegaMinNx);
}
inline bool prolong_before_sweep(const Dims& d, size_t elem, int nu2) { return restrict_after_sweep(d, elem, nu2); }

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

__device__ __forceinline__ float mul_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_t(double a, double b) { return __dmul_rn(a, b); }

// Gauss-Seidel value (S - b / n^2) / c. The product is rounded here: where the
// value is a term of another sum the compiler would fuse it into that addition,
// and a value formed twice would not have the same bits.
template <typename T>
__device__ __forceinline__ T gs_value(T S, T b, T inv, T rc) {
    return mul_t(fma_t(-b, inv, S), rc);
}

// FP32 sweeps may be over-relaxed, FP64 ones are plain: the test and the two
// operations, left to the compiler, were executed and selected from, three of ten
// FP64 instructions per cell.
template <typename T>
__device__ __forceinline__ T over_relaxed(T v, T old, T omega) {
    if (sizeof(T) == sizeof(float) && omega != T(1)) v = v + (omega - T(1)) * (v - old);
    return v;
}

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
// x sum of one row of four taps after a Gauss-Seidel sweep that ended with the
// black colour (restrict_after_sweep below): the red taps alone, at the odd
// columns 2 xc - 1 and 2 xc + 1 (odd) or the even ones. The black taps being
// exact zeros, the bits of full4.
template <typename T, typename G>
__device__ __forceinline__ T red_row(bool odd, G get) {
    return fma_t(T(3), odd ? get(2) : get(1), odd ? get(0) : get(3));
}
// the weighted sum over the planes' and rows' x sums row(kz, ky): y, then z
template <typename T, typename R>
__device__ __forceinline__ T restrict_rows(R row) {
    T p[4];
#pragma unroll
    for (int kz = 0; kz < 4; ++kz) p[kz] = full4<T>(row(kz, 0), row(kz, 1), row(kz, 2), row(kz, 3));
    return full4<T>(p[0], p[1], p[2], p[3]) * T(1.0 / 512.0);
}
// src/mg/solver.h:153-181: taps get(kz, ky, kx)
template <typename T, typename G>
__device__ __forceinline__ T restrict_taps(G get) {
    T p[4];
#pragma unroll
    for (int kz = 0; kz < 4; ++kz) p[kz] = restrict_plane<T>([&](int ky, int kx) { return get(kz, ky, kx); });
    return full4<T>(p[0], p[1], p[2], p[3]) * T(1.0 / 512.0);
}

// Column (0: odd x, 1: even x) of the black cell among the two of a row, by the
// row's y and plane's z (0: odd, 1: even); -1 for both cells (all colours).
__device__ __forceinline__ int black_col(bool black, int ry, int rz) { return black ? (ry == rz ? 0 : 1) : -1; }

// src/mg/solver.h:71-151. One fine plane of a coarse cell and its +1
// neighbours: n** on the near coarse plane, f** on the far one, second letter
// b, u along y and third l, r along x. put(rx, ry, value, scale): the fine cell
// nearest to corner (rx, ry), rx = 0 at odd x and ry = 0 at odd y, takes
// scale * value; with black only the black cells of the plane (rz = 0: odd z).
template <typename T, typename P>
__device__ __forceinline__ void prolong_row(T l, T r, T scale, int col, P put) {
    if (col < 0) {
        put(0, near4(l, r), scale);
        put(1, near4(r, l), scale);
    } else {
        put(col, near4(col ? r : l, col ? l : r), scale);
    }
}
template <typename T, typename P>
__device__ __forceinline__ void prolong_plane4(T nbl, T nbr, T nul, T nur, T fbl, T fbr, T ful, T fur, bool black,
                                               int rz, P put) {
    const T bl = near4(nbl, fbl), br = near4(nbr, fbr), ul = near4(nul, ful), ur = near4(nur, fur);  // z
    const T s = T(1.0 / 64.0);
    prolong_row(near4(bl, ul), near4(br, ur), s, black_col(black, 0, rz), [&](int rx, T v, T sc) { put(rx, 0, v, sc); });
    prolong_row(near4(ul, bl), near4(ur, br), s, black_col(black, 1, rz), [&](int rx, T v, T sc) { put(rx, 1, v, sc); });
}
// The two fine cells of a channel wall row (no y neighbour; near and far coarse
// planes), or of a row of a 2D grid (near and far coarse rows in y): near row n,
// far row f; col as black_col gives it.
template <typename T, typename P>
__device__ __forceinline__ void prolong_row2(T nl, T nr, T fl, T fr, int col, P put) {
    prolong_row(near4(nl, fl), near4(nr, fr), T(1.0 / 16.0), col, put);
}

}  // namespace afmib
