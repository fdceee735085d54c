// Geometric multigrid pieces for the pressure projection (src/mg/solver.h,
// src/mg/laplacian.h): red-black Gauss–Seidel in place of the reference's
// lexicographic CSR sweep, the reference's full-weighting restriction and
// trilinear prolongation, and a one-block CG for the coarsest level.
#include <cooperative_groups.h>

#include "dfloat.cuh"
#include "kernels.h"
#include "mg_cells.cuh"

namespace afmib {

namespace {

constexpr int BX = 32, BY = 8;
inline dim3 grid3(const Dims& d) { return dim3((d.nx + BX - 1) / BX, (d.ny + BY - 1) / BY, d.nz); }

// Per-level constants and per-row coefficients of the pressure Laplacian. The
// FP64 pipe issues one warp instruction per 16-19 clocks on an SM, conversions,
// comparisons and divisions included, so n^2 and 1/n^2 come in as kernel
// arguments, the neighbour count stays an integer and its coefficients are
// selected constants (128^3 FP64 colour 24.9 -> 22.9 us, general 104^3 27.0 -> 20.8; with them formed per
// thread a cell cost 10 FP64 instructions instead of the update's 7).
template <typename T>
struct LapK {
    T off, inv;  // n^2, 1 / n^2
};
template <typename T>
inline LapK<T> lap_k(const Dims& d) {
    return LapK<T>{T(d.n) * T(d.n), T(1) / (T(d.n) * T(d.n))};
}
// the row's neighbour count (6; 5 or 4 at channel walls; 4 in 2D) and its reciprocal
template <typename T>
__device__ __forceinline__ T lap_count(int c) {
    return c == 6 ? T(6) : (c == 5 ? T(5) : T(4));
}
template <typename T>
__device__ __forceinline__ T lap_rcount(int c) {
    return c == 6 ? T(1.0 / 6.0) : (c == 5 ? T(1.0 / 5.0) : T(0.25));
}


// Neighbour sum and diagonal factor of the Laplacian row at (x, y, z):
// L x = n^2 * (S - c * x_i), c = 6 in the interior and one less per channel
// wall (Neumann, src/mg/laplacian.h:75-82). A one-cell z extent (2D) folds
// its two self-neighbours into the diagonal, src/mg/laplacian.h:62-73.
template <typename T>
__device__ __forceinline__ void lap_row(const Dims& d, const T* x, int xi, int yi, int zi, T& S, int& c) {
    if (d.nz == 1) {
        S = x[lin(d, xm1(d, xi), yi, zi)] + x[lin(d, xp1(d, xi), yi, zi)];
        c = 4;
    } else {
        S = (x[lin(d, xm1(d, xi), yi, zi)] + x[lin(d, xp1(d, xi), yi, zi)]) +
            (x[lin(d, xi, yi, zm1(d, zi))] + x[lin(d, xi, yi, zp1(d, zi))]);
        c = 6;
    }
    if (d.channel) {
        if (yi > 0) S += x[lin(d, xi, yi - 1, zi)]; else --c;
        if (yi < d.ny - 1) S += x[lin(d, xi, yi + 1, zi)]; else --c;
    } else {
        S += x[lin(d, xi, ym1(d, yi), zi)] + x[lin(d, xi, yp1(d, yi), zi)];
    }
}

// Neighbour sum and diagonal factor of lap_row with Ix2 or IxG indexing (same
// terms, same order).
template <typename T, typename IX>
__device__ __forceinline__ void lap_row2(const Dims& d, const IX& I, const T* x, int xi, int yi, int zi,
                                         T& S, int& c) {
    if (d.nz == 1) {
        S = x[I.at(I.xm(xi), yi, zi)] + x[I.at(I.xp(xi), yi, zi)];
        c = 4;
    } else {
        S = (x[I.at(I.xm(xi), yi, zi)] + x[I.at(I.xp(xi), yi, zi)]) + (x[I.at(xi, yi, I.zm(zi))] + x[I.at(xi, yi, I.zp(zi))]);
        c = 6;
    }
    if (d.channel) {
        if (yi > 0) S += x[I.at(xi, yi - 1, zi)]; else --c;
        if (yi < d.ny - 1) S += x[I.at(xi, yi + 1, zi)]; else --c;
    } else {
        S += x[I.at(xi, I.ym(yi), zi)] + x[I.at(xi, I.yp(yi), zi)];
    }
}

template <typename T, typename IX>
__global__ void k_lap(Dims d, LapK<T> k, T* __restrict__ out, const T* __restrict__ in) {
    wait_launch();
    const int x = blockIdx.x * BX + threadIdx.x, y = blockIdx.y * BY + threadIdx.y, z = blockIdx.z;
    if (x >= d.nx || y >= d.ny) return;
    const IX I(d);
    T S;
    int c;
    lap_row2(d, I, in, x, y, z, S, c);
    const int i = I.at(x, y, z);
    out[i] = k.off * (S - lap_count<T>(c) * in[i]);
}

template <typename T, typename IX>
__global__ void k_residual(Dims d, LapK<T> k, T* __restrict__ r, const T* __restrict__ xv, const T* __restrict__ b) {
    wait_launch();
    const int x = blockIdx.x * BX + threadIdx.x, y = blockIdx.y * BY + threadIdx.y, z = blockIdx.z;
    if (x >= d.nx || y >= d.ny) return;
    const IX I(d);
    T S;
    int c;
    lap_row2(d, I, xv, x, y, z, S, c);
    const int i = I.at(x, y, z);
    r[i] = b[i] - k.off * (S - lap_count<T>(c) * xv[i]);
}

template <typename T, typename IX>
__global__ void __launch_bounds__(kRedBlock) k_residual_norm(Dims d, LapK<T> k, T* __restrict__ r,
                                                            const T* __restrict__ xv, const T* __restrict__ b,
                                                            RedScratch sc, double* out) {
    wait_launch();
    const int xi = blockIdx.x * kRBX + threadIdx.x, yi = blockIdx.y * kRBY + threadIdx.y;
    const IX I(d);
    T acc = T(0);
    if (xi < d.nx && yi < d.ny)
#pragma unroll 2
        for (int zi = blockIdx.z; zi < d.nz; zi += gridDim.z) {
            T S;
            int c;
            lap_row2(d, I, xv, xi, yi, zi, S, c);
            const int i = I.at(xi, yi, zi);
            const T ri = b[i] - k.off * (S - lap_count<T>(c) * xv[i]);
            r[i] = ri;
            acc += ri * ri;
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// Mixed form: defect of the FP64 potential, r = b - L x evaluated in FP64 and
// stored in TD for the FP32 inner V-cycles; out[0] = r.r.
// r_lo: also the rest of the FP64 residual, float(r - r_float), the second
// word of the double-float pair that k_lap_update_df updates.
template <typename TD>
__global__ void __launch_bounds__(kRedBlock) k_lap_defect(Dims d, LapK<double> k, TD* __restrict__ r,
                                                         const double* __restrict__ xv,
                                                         const double* __restrict__ b, RedScratch sc, double* out,
                                                         float* __restrict__ r_lo, bool lo_split) {
    wait_launch();
    const int xi = blockIdx.x * kRBX + threadIdx.x, yi = blockIdx.y * kRBY + threadIdx.y;
    TD acc = TD(0);
    if (xi < d.nx && yi < d.ny)
#pragma unroll 2
        for (int zi = blockIdx.z; zi < d.nz; zi += gridDim.z) {
            double S;
            int c;
            lap_row(d, xv, xi, yi, zi, S, c);
            const long long i = lin(d, xi, yi, zi);
            float lo;
            const TD ri = defect_words(b[i] - k.off * (S - lap_count<double>(c) * xv[i]), r_lo ? &lo : nullptr, lo_split);
            r[i] = ri;
            if (r_lo) r_lo[i] = lo;
            acc += ri * ri;
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// Mixed form: the first defect of a pressure solve in double-float on the
// FP32 pipe (the FP64 kernel is FP64-pipe bound: 81% busy, ncu), with the
// mean removal of b folded in: r = (b - m) - n^2 (S - c x0), m = sum * scale
// (the FP64 form's k_sub_scalar value; sum null: m = 0). The neighbours of an axis
// are added in FP64, the sums, x0 and b split by integer operations (df_split), the
// sums over the axes, c x0 and the n^2 scaling are pairs: three FP64 additions and
// five splits per cell, two z cells' loads first: 178 us at 256^3 (eight splits cell
// by cell: 282; four cells: 223). The pair is the FP32 defect rh and its rest rl of
// k_lap_update_df, out[0] = rh.rh.
template <int ZU, typename IX, bool SPLIT>
__global__ void __launch_bounds__(kRedBlock) k_lap_defect_df(Dims d, float* __restrict__ rh, float* __restrict__ rl,
                                                            const double* __restrict__ xv,
                                                            const double* __restrict__ b, const double* sum,
                                                            double scale, RedScratch sc, double* out) {
    wait_launch();
    const IX I(d);
    const typename RowIx<IX, SPLIT>::type E(d);  // of rh
    const int x = blockIdx.x * kRBX + threadIdx.x, y = blockIdx.y * kRBY + threadIdx.y;
    const df2 off = {float(d.n) * float(d.n), 0.f};  // exact for n < 4096
    const df2 m = sum ? df_split(sum[0] * scale) : df2{0.f, 0.f};
    const bool lo = !d.channel || y > 0, hi = !d.channel || y < d.ny - 1;
    const float c = (d.nz > 1 ? 6.f : 4.f) - (lo ? 0.f : 1.f) - (hi ? 0.f : 1.f);
    float acc = 0.f;
    if (x < d.nx && y < d.ny)
        for (int zb = blockIdx.z; zb < d.nz / ZU; zb += gridDim.z) {
            // every load of the batch first
            const int z0 = zb * ZU;
            double col[ZU + 2], x0[ZU], x1[ZU], y0[ZU], y1[ZU], bv[ZU];
#pragma unroll
            for (int k = 0; k < ZU + 2; ++k) col[k] = xv[I.at(x, y, I.wz(z0 + k - 1))];
#pragma unroll
            for (int k = 0; k < ZU; ++k) {
                const int z = z0 + k;
                x0[k] = xv[I.at(I.xm(x), y, z)];
                x1[k] = xv[I.at(I.xp(x), y, z)];
                y0[k] = lo ? xv[I.at(x, I.ym(y), z)] : 0.0;
                y1[k] = hi ? xv[I.at(x, I.yp(y), z)] : 0.0;
                bv[k] = b[I.at(x, y, z)];
            }
#pragma unroll
            for (int k = 0; k < ZU; ++k) {
                df2 S = df_split(x0[k] + x1[k]);
                if (d.nz > 1) S = df_add(S, df_split(col[k] + col[k + 2]));
                S = df_add(S, df_split(y0[k] + y1[k]));
                const df2 L = df_mul(off, df_add(S, df_neg(df_mul(df2{c, 0.f}, df_split(col[k + 1])))));
                const df2 r = df_add(df_add(df_split(bv[k]), df_neg(m)), df_neg(L));
                const int i = I.at(x, y, z0 + k);
                rh[E.at(x, y, z0 + k)] = r.hi;
                rl[i] = r.lo;
                acc += r.hi * r.hi;
            }
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// Mixed form, recursive outer residual of the pressure solve: with the FP32
// correction e of the inner V-cycles, x += e (FP64) and the residual, kept
// as a double-float pair (rh: the FP32 right-hand side of the V-cycles, rl:
// the rest), loses L e evaluated in double-float (df_lap_row); out[0] =
// rh.rh, as the FP64 defect's norm.
__global__ void __launch_bounds__(kRedBlock) k_lap_update_df(Dims d, double* __restrict__ x,
                                                            const float* __restrict__ e, float* __restrict__ rh,
                                                            float* __restrict__ rl, RedScratch sc, double* out) {
    wait_launch();
    const int xi = blockIdx.x * kRBX + threadIdx.x, yi = blockIdx.y * kRBY + threadIdx.y;
    const float off = float(d.n) * float(d.n);
    float acc = 0.f;
    if (xi < d.nx && yi < d.ny)
        for (int zi = blockIdx.z; zi < d.nz; zi += gridDim.z) {
            const long long i = lin(d, xi, yi, zi);
            const float e0 = e[i];
            float nb[6];
            int m = 0;
            nb[m++] = e[lin(d, xm1(d, xi), yi, zi)];
            nb[m++] = e[lin(d, xp1(d, xi), yi, zi)];
            if (d.nz > 1) {
                nb[m++] = e[lin(d, xi, yi, zm1(d, zi))];
                nb[m++] = e[lin(d, xi, yi, zp1(d, zi))];
            }
            float c = d.nz > 1 ? 6.f : 4.f;
            if (d.channel) {
                if (yi > 0) nb[m++] = e[lin(d, xi, yi - 1, zi)]; else c -= 1.f;
                if (yi < d.ny - 1) nb[m++] = e[lin(d, xi, yi + 1, zi)]; else c -= 1.f;
            } else {
                nb[m++] = e[lin(d, xi, ym1(d, yi), zi)];
                nb[m++] = e[lin(d, xi, yp1(d, yi), zi)];
            }
            for (int j = m; j < 6; ++j) nb[j] = 0.f;
            const df2 le = df_lap_row(e0, nb, 6, c, off);
            df2 r;
            r.hi = rh[i];
            r.lo = rl[i];
            r = df_add(r, df_neg(le));
            rh[i] = r.hi;
            rl[i] = r.lo;
            x[i] = x[i] + cvt<double, float>(e0);
            acc += r.hi * r.hi;
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// The same on 3D grids with nz % ZU == 0, two z cells per thread with every load
// of the pair issued first (as k_helm_update_df2); the same rows, so the
// same bits.
template <int ZU, int MINB, typename IX, bool SPLIT>
__global__ void __launch_bounds__(kRedBlock, MINB) k_lap_update_df2(Dims d, double* __restrict__ x,
                                                             const float* __restrict__ e, float* __restrict__ rh,
                                                             float* __restrict__ rl, RedScratch sc, double* out) {
    wait_launch();
    const IX I(d);
    const typename RowIx<IX, SPLIT>::type E(d);  // of e and rh
    const int xi = blockIdx.x * kRBX + threadIdx.x, yi = blockIdx.y * kRBY + threadIdx.y;
    const float off = float(d.n) * float(d.n);
    const bool has_ym = !d.channel || yi > 0, has_yp = !d.channel || yi < d.ny - 1;
    const float c = 6.f - (has_ym ? 0.f : 1.f) - (has_yp ? 0.f : 1.f);
    const int ym = I.ym(yi), yp = I.yp(yi);
    float acc = 0.f;
    if (xi < d.nx && yi < d.ny)
        for (int zb = blockIdx.z; zb < d.nz / ZU; zb += gridDim.z) {
            const int z0 = zb * ZU;
            float col[ZU + 2], ex0[ZU], ex1[ZU], ey0[ZU], ey1[ZU], h[ZU], l[ZU];
            double xv[ZU];
#pragma unroll
            for (int u = 0; u < ZU + 2; ++u) col[u] = e[E.at(xi, yi, I.wz(z0 + u - 1))];  // z0 - 1 .. z0 + ZU
#pragma unroll
            for (int u = 0; u < ZU; ++u) {
                const int z = z0 + u, i = I.at(xi, yi, z);
                ex0[u] = e[E.at(I.xm(xi), yi, z)];
                ex1[u] = e[E.at(I.xp(xi), yi, z)];
                ey0[u] = has_ym ? e[E.at(xi, ym, z)] : 0.f;
                ey1[u] = has_yp ? e[E.at(xi, yp, z)] : 0.f;
                h[u] = rh[E.at(xi, yi, z)];
                l[u] = rl[i];
                xv[u] = x[i];
            }
#pragma unroll
            for (int u = 0; u < ZU; ++u) {
                const int i = I.at(xi, yi, z0 + u);
                const float e0 = col[u + 1];
                // the general kernel's neighbour order: x, z, then the y neighbours present
                float nb[6] = {ex0[u], ex1[u], col[u], col[u + 2], has_ym ? ey0[u] : ey1[u], has_ym ? ey1[u] : 0.f};
                if (!has_yp) nb[5] = 0.f;
                const df2 le = df_lap_row(e0, nb, 6, c, off);
                df2 r;
                r.hi = h[u];
                r.lo = l[u];
                r = df_add(r, df_neg(le));
                rh[E.at(xi, yi, z0 + u)] = r.hi;
                rl[i] = r.lo;
                x[i] = xv[u] + cvt<double, float>(e0);
                acc += r.hi * r.hi;
            }
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// The same defect without FP64 instructions (lap_residual_bfp): with
// n^2 = 2^k2, b 2^-k2 - sum(nb) + c x0 is formed exactly in int64 at the
// cell's largest exponent and scaled back by 2^k2.
__global__ void __launch_bounds__(kRedBlock) k_lap_defect_bfp(Dims d, int k2, float* __restrict__ r,
                                                             const double* __restrict__ xv, const double* __restrict__ b,
                                                             RedScratch sc, double* out) {
    wait_launch();
    const int xi = blockIdx.x * kRBX + threadIdx.x, yi = blockIdx.y * kRBY + threadIdx.y;
    float acc = 0.f;
    if (xi < d.nx && yi < d.ny)
#pragma unroll 2
        for (int zi = blockIdx.z; zi < d.nz; zi += gridDim.z) {
            const long long i = lin(d, xi, yi, zi);
            double nb[6];
            int m = 0, c = 6;
            nb[m++] = xv[lin(d, xm1(d, xi), yi, zi)];
            nb[m++] = xv[lin(d, xp1(d, xi), yi, zi)];
            if (d.nz == 1) {
                c = 4;
            } else {
                nb[m++] = xv[lin(d, xi, yi, zm1(d, zi))];
                nb[m++] = xv[lin(d, xi, yi, zp1(d, zi))];
            }
            if (d.channel) {
                if (yi > 0) nb[m++] = xv[lin(d, xi, yi - 1, zi)]; else --c;
                if (yi < d.ny - 1) nb[m++] = xv[lin(d, xi, yi + 1, zi)]; else --c;
            } else {
                nb[m++] = xv[lin(d, xi, ym1(d, yi), zi)];
                nb[m++] = xv[lin(d, xi, yp1(d, yi), zi)];
            }
            const float ri = lap_residual_bfp(b[i], xv[i], nb, m, c, k2);
            r[i] = ri;
            acc += ri * ri;
        }
    double a[1] = {(double)acc};
    grid_sum<1>(a, sc, out);
}

// One colour of red-black Gauss–Seidel: x_i = (b_i - n^2 S) / (-c n^2).
// omega != 1: over-relaxed update x + omega (gs - x); omega == 1 is plain
// Gauss-Seidel, bit for bit
template <typename T, typename IX>
__global__ void k_rbgs(Dims d, LapK<T> k, int color, T omega, T* __restrict__ xv, const T* __restrict__ b) {
    wait_launch();
    const int y = blockIdx.y * BY + threadIdx.y, z = blockIdx.z;
    const int x = 2 * (blockIdx.x * BX + threadIdx.x) + ((y + z + color) & 1);
    if (x >= d.nx || y >= d.ny) return;
    const IX I(d);
    T S;
    int c;
    lap_row2(d, I, xv, x, y, z, S, c);
    const int i = I.at(x, y, z);
    T v = (S - b[i] * k.inv) * lap_rcount<T>(c);
    xv[i] = sizeof(T) == sizeof(float) ? over_relaxed(v, xv[i], omega) : v;
}

// Batched forms: each thread takes ZU cells along z of its (x, y) column and
// computes all of them before storing any, so that ZU cells' loads are in
// flight at once (on GB300 one cell per thread leaves the stencil bound by
// block turnover, near 3 TB/s). Within one colour the red cells read only
// black ones, so the delayed stores change nothing: same values as the
// one-cell kernels.
constexpr int kZU = 8;  // z cells per thread of the batched stencil kernels
constexpr int kZU32 = 4;  // ... of the FP32 red-black colour
constexpr int kZU64 = 2;  // ... of the FP64 one: 22.9 us per 128^3 colour with 8 (512 blocks), 20.9 with 4, 20.8 with 2, 20.4 with 1

template <typename T, int ZU, typename IX>
__device__ __forceinline__ void rbgs_z2_body(Dims d, const LapK<T>& k, int color, T omega, T* __restrict__ xv,
                                             const T* __restrict__ b, int rev) {
    const IX I(d);
    const uint3 B = block_at(rev);
    const int y = B.y * BY + threadIdx.y, t = B.x * BX + threadIdx.x, z0 = B.z * ZU;
    if (y >= d.ny || 2 * t >= d.nx) return;
    T val[ZU];
    int at[ZU];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int z = z0 + u, x = 2 * t + ((y + z + color) & 1);
        T S;
        int c;
        lap_row2(d, I, xv, x, y, z, S, c);
        const int i = I.at(x, y, z);
        val[u] = (S - b[i] * k.inv) * lap_rcount<T>(c);
        if (sizeof(T) == sizeof(float)) val[u] = over_relaxed(val[u], xv[i], omega);
        at[u] = i;
    }
#pragma unroll
    for (int u = 0; u < ZU; ++u) xv[at[u]] = val[u];
}
template <typename T, int ZU, typename IX>
__global__ void k_rbgs_z2(Dims d, LapK<T> k, int color, T omega, T* __restrict__ xv, const T* __restrict__ b, int rev) {
    wait_launch();
    rbgs_z2_body<T, ZU, IX>(d, k, color, omega, xv, b, rev);
}

// A whole sweep from x = 0 in one pass: b is read, x written, x never read. A red
// cell's update has the neighbour sum zero, so the reds that a black cell sums are
// formed from b on the fly. A thread owns the pairs (2t, 2t+1) of its (y, z)
// column, one red and one black cell each; of the black cell's six reds one is the
// pair's own, the two along z are the own reds of the pairs above and below, and
// the other three are formed again (a fifth load each of b, from L1). `zero` is a
// kernel argument, so that the arithmetic is rbgs_z2_body's and not a folded
// constant (nor its products fused: gs_value): the same bits as a memset of x and
// the two colours. With the viscous
// solves' first sweeps in the same form: IB steps of the mixed form at 256^3 16.20
// -> 15.77 ms, at 96x80x112 3.88 -> 3.74; FP64 steps unchanged (13.8 ms at 128^3:
// the reds formed again cost the FP64 pipe what the launch saves).
template <typename T, int ZU, int MINB, typename IX, bool SPLIT = false>
__global__ void __launch_bounds__(BX * BY, MINB) k_rbgs_first(Dims d, LapK<T> k, T omega, T* __restrict__ xv,
                                                             const T* __restrict__ b, int rev, T zero) {
    wait_launch();
    const IX I(d);
    const typename RowIx<IX, SPLIT>::type E(d);
    const uint3 B = block_at(rev);
    const int y = B.y * BY + threadIdx.y, t = B.x * BX + threadIdx.x, z0 = B.z * ZU;
    if (y >= d.ny || 2 * t >= d.nx) return;
    const bool flat = d.nz == 1;
    auto count = [&](int yy) {
        int c = flat ? 4 : 6;
        if (d.channel) {
            if (!(yy > 0)) --c;
            if (!(yy < d.ny - 1)) --c;
        }
        return c;
    };
    auto update = [&](T S, int i, int c) {
        T v = gs_value(S, b[i], k.inv, lap_rcount<T>(c));
        return over_relaxed(v, zero, omega);
    };
    const int c = count(y);
    const bool lo = !d.channel || y > 0, hi = !d.channel || y < d.ny - 1;
    const int ylo = I.ym(y), yhi = I.yp(y), clo = count(ylo), chi = count(yhi);
    // own reds of planes z0 - 1 ... z0 + ZU
    T red[ZU + 2];
#pragma unroll
    for (int u = 0; u < ZU + 2; ++u) {
        const int z = z0 + u - 1;
        red[u] = flat && u != 1 ? zero : update(zero, E.at(2 * t + ((y + z) & 1), y, I.wz(z)), c);
    }
    T val[ZU];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int z = z0 + u, p = (y + z) & 1, x = 2 * t + 1 - p;
        T S = red[u + 1] + update(zero, E.at(p ? I.xm(2 * t) : I.xp(2 * t + 1), y, z), c);
        if (!flat) S = S + (red[u] + red[u + 2]);
        if (d.channel) {
            if (lo) S += update(zero, E.at(x, ylo, z), clo);
            if (hi) S += update(zero, E.at(x, yhi, z), chi);
        } else {
            S += update(zero, E.at(x, ylo, z), clo) + update(zero, E.at(x, yhi, z), chi);
        }
        val[u] = update(S, E.at(x, y, z), c);
    }
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int z = z0 + u, p = (y + z) & 1;
        xv[E.at(2 * t + p, y, z)] = red[u + 1];
        xv[E.at(2 * t + 1 - p, y, z)] = val[u];
    }
}
// One colour with x and b split by colour within each row (Split2): every load and
// store of a warp is 32 consecutive words, the z neighbours come from the column's
// registers (mg_split_ok for what it measured).
template <int ZU, int MINB>
__global__ void __launch_bounds__(BX * BY, MINB) k_rbgs_split(Dims d, LapK<float> k, int color, float omega,
                                                             float* __restrict__ xv, const float* __restrict__ b,
                                                             int rev) {
    wait_launch();
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int y = B.y * BY + threadIdx.y, t = B.x * BX + threadIdx.x, z0 = B.z * ZU, h = d.nx / 2;
    const bool lo = !d.channel || y > 0, hi = !d.channel || y < d.ny - 1;
    const int c = 6 - (lo ? 0 : 1) - (hi ? 0 : 1);
    const int yo = y << I.lx, ym = I.ym(y) << I.lx, yp = I.yp(y) << I.lx;
    const int other = (1 - color) * h + t, own = color * h + t;
    float o[ZU + 2], side[ZU], dn[ZU], up[ZU], bv[ZU], old[ZU];
#pragma unroll
    for (int u = 0; u < ZU + 2; ++u) o[u] = xv[(I.wz(z0 + u - 1) << I.lxy) + yo + other];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int zo = (z0 + u) << I.lxy;
        // the cell is x = 2t + p: beside it the pair's other cell and one of the next or last pair
        const int p = (y + z0 + u + color) & 1, tn = (p ? t + 1 : t - 1) & (h - 1);
        side[u] = xv[zo + yo + other - t + tn];
        dn[u] = lo ? xv[zo + ym + other] : 0.f;
        up[u] = hi ? xv[zo + yp + other] : 0.f;
        bv[u] = b[zo + yo + own];
        old[u] = xv[zo + yo + own];
    }
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        float S = (o[u + 1] + side[u]) + (o[u] + o[u + 2]);
        if (d.channel) {
            if (lo) S += dn[u];
            if (hi) S += up[u];
        } else {
            S += dn[u] + up[u];
        }
        xv[((z0 + u) << I.lxy) + yo + own] = over_relaxed(gs_value(S, bv[u], k.inv, lap_rcount<float>(c)), old[u], omega);
    }
}

template <typename T, int ZU, int MINB, typename IX>
__global__ void __launch_bounds__(BX * BY, MINB) k_rbgs_z2b(Dims d, LapK<T> k, int color, T omega, T* __restrict__ xv,
                                                           const T* __restrict__ b, int rev) {
    wait_launch();
    rbgs_z2_body<T, ZU, IX>(d, k, color, omega, xv, b, rev);
}

// The FP32 colour on float pairs: a thread owns the pairs (2t, 2t+1) of its
// (y, z) column, one cell of each pair being the colour's. Per ZU-cell
// column it loads ZU + 2 pairs of its own column (the z neighbours come from
// the same registers), the pairs of the rows y - 1 and y + 1, and the pairs
// of b: 4.25 eight-byte loads per updated cell, each warp instruction reading
// 256 contiguous bytes, against the scalar kernel's eight stride-2 loads. The
// x neighbour across the pair boundary comes from the adjacent lane by a
// shuffle (the first and last lanes load it). The colour is uniform across a
// warp (its lanes share y and z). The update is rbgs_z2_body's arithmetic in
// the same order, so the same bits; the pair is stored whole, the other
// colour's value unchanged (no thread writes that colour in this launch).
template <int ZU, int MINB>
__global__ void __launch_bounds__(BX * BY, MINB) k_rbgs_pair(Dims d, int color, float omega, float* __restrict__ xv,
                                                            const float* __restrict__ b, int rev) {
    wait_launch();
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int t = B.x * BX + threadIdx.x, y = B.y * BY + threadIdx.y, z0 = B.z * ZU;
    const float2* __restrict__ xp = reinterpret_cast<const float2*>(xv);
    const float2* __restrict__ bp = reinterpret_cast<const float2*>(b);
    auto pr = [&](int yy, int zz) { return I.at(2 * t, yy, zz) >> 1; };
    const bool has_lo = !d.channel || y > 0, has_hi = !d.channel || y < d.ny - 1;
    const int ylo = d.channel ? y - 1 : I.ym(y), yhi = d.channel ? y + 1 : I.yp(y);
    float2 col[ZU + 2], ly[ZU], hy[ZU], bb[ZU];
#pragma unroll
    for (int k = 0; k < ZU + 2; ++k) col[k] = xp[pr(y, (z0 - 1 + k) & I.mz)];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        ly[u] = has_lo ? xp[pr(ylo, z0 + u)] : make_float2(0.f, 0.f);
        hy[u] = has_hi ? xp[pr(yhi, z0 + u)] : make_float2(0.f, 0.f);
        bb[u] = bp[pr(y, z0 + u)];
    }
    const float inv = 1.f / (float(d.n) * float(d.n));
    float2 out[ZU];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int z = z0 + u, p = (y + z + color) & 1;
        const float2 self = col[u + 1];
        float left, right;
        if (p == 0) {  // the cell 2t: its left neighbour is the previous pair's second value
            float prev = __shfl_up_sync(0xffffffffu, self.y, 1);
            if (threadIdx.x == 0) prev = xv[I.at((2 * t - 1) & I.mx, y, z)];
            left = prev;
            right = self.y;
        } else {  // the cell 2t + 1: its right neighbour is the next pair's first value
            float next = __shfl_down_sync(0xffffffffu, self.x, 1);
            if (threadIdx.x == BX - 1) next = xv[I.at((2 * t + 2) & I.mx, y, z)];
            left = self.x;
            right = next;
        }
        const float zm = p ? col[u].y : col[u].x, zq = p ? col[u + 2].y : col[u + 2].x;
        float S = (left + right) + (zm + zq), c = 6.f;
        const float yl = p ? ly[u].y : ly[u].x, yh = p ? hy[u].y : hy[u].x;
        if (d.channel) {
            if (has_lo) S += yl; else c -= 1.f;
            if (has_hi) S += yh; else c -= 1.f;
        } else {
            S += yl + yh;
        }
        const float rc = (c == 6.f) ? float(1.0 / 6.0) : ((c == 5.f) ? float(1.0 / 5.0) : (c == 4.f ? 0.25f : 1.f / c));
        const float bi = p ? bb[u].y : bb[u].x;
        float v = (S - bi * inv) * rc;
        if (omega != 1.f) v = v + (omega - 1.f) * (v - (p ? self.y : self.x));
        out[u] = p ? make_float2(self.x, v) : make_float2(v, self.y);
    }
    float2* __restrict__ xw = reinterpret_cast<float2*>(xv);
#pragma unroll
    for (int u = 0; u < ZU; ++u) xw[pr(y, z0 + u)] = out[u];
}

template <typename T, int ZU, typename IX>
__global__ void k_residual_z2(Dims d, LapK<T> k, T* __restrict__ r, const T* __restrict__ xv, const T* __restrict__ b,
                              int rev) {
    wait_launch();
    const IX I(d);
    const uint3 B = block_at(rev);
    const int x = B.x * BX + threadIdx.x, y = B.y * BY + threadIdx.y, z0 = B.z * ZU;
    if (x >= d.nx || y >= d.ny) return;
    T val[ZU];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        T S;
        int c;
        lap_row2(d, I, xv, x, y, z0 + u, S, c);
        const int i = I.at(x, y, z0 + u);
        val[u] = b[i] - k.off * (S - lap_count<T>(c) * xv[i]);
    }
#pragma unroll
    for (int u = 0; u < ZU; ++u) r[I.at(x, y, z0 + u)] = val[u];
}

// The residual on the red cells alone (restrict_after_sweep): the same
// expression; the black cells of r are not written. ZU cells along z per thread.
template <typename T, int ZU, typename IX>
__global__ void k_residual_red(Dims d, LapK<T> k, T* __restrict__ r, const T* __restrict__ xv, const T* __restrict__ b,
                               int rev) {
    wait_launch();
    const IX I(d);
    const uint3 B = block_at(rev);
    const int t = B.x * BX + threadIdx.x, y = B.y * BY + threadIdx.y, z0 = B.z * ZU;
    if (2 * t >= d.nx || y >= d.ny) return;
    T val[ZU];
    int at[ZU];
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int z = z0 + u, x = 2 * t + ((y + z) & 1);
        T S;
        int c;
        lap_row2(d, I, xv, x, y, z, S, c);
        const int i = I.at(x, y, z);
        val[u] = b[i] - k.off * (S - lap_count<T>(c) * xv[i]);
        at[u] = i;
    }
#pragma unroll
    for (int u = 0; u < ZU; ++u) r[at[u]] = val[u];
}

// ---------------------------------------------------------------------------
// Pipelined red-black sweep: one full sweep (red, then black) per launch, out
// of place (xin -> xout). A block owns FY full-width rows (every x of the row,
// so there is no x halo: x wraps inside shared memory) and a chunk of ZC
// planes, and marches along z. At step k it updates the red cells of plane k
// on the rows tile +- 1, then the black cells of plane k-1 on the tile, then
// writes plane k-1 of the tile. Rows of x (tile +- 2) and of b (tile +- 1)
// arrive in a ring of R = D + 4 plane slots by asynchronous 16-byte copies
// (cp.async) that all threads issue D planes ahead, one commit group per
// plane, so the march does not wait on DRAM. The blocks are persistent and
// take (row strip, z chunk) items in order. Every update is the per-colour
// kernel's arithmetic with the same terms in the same order, so a pipelined
// sweep equals the two per-colour launches cell for cell.
// ---------------------------------------------------------------------------
namespace pipe {
__device__ __forceinline__ unsigned saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_pending() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
}  // namespace pipe

constexpr int kPipeThreads = 256;

// Gauss-Seidel value of one cell from its six neighbours and b, the
// per-colour kernel's arithmetic (rbgs_cell) in the same order.
template <typename T, bool CH>
__device__ __forceinline__ T gs_value(T xm, T xp, T zm, T zp, T ym, T yp, T bv, T inv, int gy, int ny) {
    T S = (xm + xp) + (zm + zp);
    T c = T(6);
    if (CH) {
        if (gy > 0) S += ym; else c -= T(1);
        if (gy < ny - 1) S += yp; else c -= T(1);
    } else {
        S += ym + yp;
    }
    const T rc = (c == T(6)) ? T(1.0 / 6.0) : ((c == T(5)) ? T(1.0 / 5.0) : (c == T(4) ? T(0.25) : T(1) / c));
    return (S - bv * inv) * rc;
}

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    typedef float4 type;
};
template <>
struct Vec4<double> {
    typedef double4 type;
};

// One colour of one plane row segment by quads: the quad of four cells at
// x = 4q .. 4q+3 holds two cells of the colour, at offsets par and par + 2.
template <typename T, bool CH>
__device__ __forceinline__ void gs_quad(T* row, const T* rowm, const T* rowp, const T* zmr, const T* zpr, const T* br,
                                        int q, int nq, int par, T inv, int gy, int ny) {
    typedef typename Vec4<T>::type V;
    V c = reinterpret_cast<V*>(row)[q];
    const V n = reinterpret_cast<const V*>(rowm)[q], s = reinterpret_cast<const V*>(rowp)[q];
    const V a = reinterpret_cast<const V*>(zmr)[q], e = reinterpret_cast<const V*>(zpr)[q];
    const V bb = reinterpret_cast<const V*>(br)[q];
    if (par == 0) {
        const T left = row[4 * (q == 0 ? nq : q) - 1];
        c.x = gs_value<T, CH>(left, c.y, a.x, e.x, n.x, s.x, bb.x, inv, gy, ny);
        c.z = gs_value<T, CH>(c.y, c.w, a.z, e.z, n.z, s.z, bb.z, inv, gy, ny);
    } else {
        const T right = row[q + 1 == nq ? 0 : 4 * (q + 1)];
        c.y = gs_value<T, CH>(c.x, c.z, a.y, e.y, n.y, s.y, bb.y, inv, gy, ny);
        c.w = gs_value<T, CH>(c.z, right, a.w, e.w, n.w, s.w, bb.w, inv, gy, ny);
    }
    reinterpret_cast<V*>(row)[q] = c;
}

// Power-of-two extents only (every level the sweep serves): indices are
// shifts and masks. CH: channel walls in y (Neumann rows, no wrap in y).
template <typename T, int D, bool CH>
__global__ void __launch_bounds__(kPipeThreads, 1) k_rbgs_pipe(Dims d, const T* __restrict__ xin, T* __restrict__ xout,
                                                            const T* __restrict__ b, int FY, int ZC, int lnx, int lny) {
    wait_launch();
    extern __shared__ __align__(128) unsigned char smem[];
    typedef typename Vec4<T>::type V;
    constexpr int R = D + 4;
    const int nx = d.nx, XR = FY + 4, BR = FY + 2;
    const int xplane = XR * nx, bplane = BR * nx;
    T* xs = (T*)smem;                 // [R][XR][nx]
    T* bs = xs + (size_t)R * xplane;  // [R][BR][nx]
    const int tid = threadIdx.x;
    const int lq = lnx - 2, nq = nx >> 2, qmask = nq - 1;  // quads per row
    const int ymask = d.ny - 1, zmask = d.nz - 1;
    const int lcpr = lnx + (sizeof(T) == 8 ? 3 : 2) - 4;  // log2 of the 16-byte chunks per row
    const int cmask = (1 << lcpr) - 1;
    const T inv = T(1) / (T(d.n) * T(d.n));
    const int nstrip = d.ny / FY, items = nstrip * (d.nz / ZC);
    int s_first = 0;
    auto next_slot = [](int q) { return q + 1 == R ? 0 : q + 1; };
    auto prev_slot = [](int q) { return q == 0 ? R - 1 : q - 1; };
    auto row_ok = [&](int gy) { return !CH || (gy >= 0 && gy < d.ny); };
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int y0 = (item % nstrip) * FY, z0 = (item / nstrip) * ZC, zend = z0 + ZC;
        const int pfirst = z0 - 2, plast = zend + 1;
        auto issue = [&](int p, int q) {
            if (p <= plast) {
                const long long zoff = (long long)(p & zmask) << lny;
                for (int c = tid; c < ((XR + BR) << lcpr); c += kPipeThreads) {
                    const int r = c >> lcpr, o = c & cmask;
                    const bool isx = r < XR;
                    const int gy = isx ? y0 - 2 + r : y0 - 1 + (r - XR);
                    if (!row_ok(gy)) continue;
                    const T* src = (isx ? xin : b) + ((zoff + (gy & ymask)) << lnx);
                    T* dst = isx ? xs + (size_t)q * xplane + (r << lnx) : bs + (size_t)q * bplane + ((r - XR) << lnx);
                    pipe::cp16((char*)dst + 16 * o, (const char*)src + 16 * o);
                }
            }
            pipe::commit();
        };
        int next = pfirst, snext = s_first;
        for (; next <= pfirst + R - 2; ++next, snext = next_slot(snext)) issue(next, snext);
        int skm1 = s_first, sk = next_slot(s_first);
        for (int k = z0 - 1; k <= zend; ++k) {
            const int skp1 = next_slot(sk), skm2 = prev_slot(skm1);
            pipe::wait_pending<D>();
            __syncthreads();
            T* const Xm = xs + (size_t)skm1 * xplane;
            T* const X0 = xs + (size_t)sk * xplane;
            T* const Xp = xs + (size_t)skp1 * xplane;
            {
                // red cells of plane k, rows tile +- 1
                const int gz = k & zmask;
                const T* B0 = bs + (size_t)sk * bplane;
                for (int e = tid; e < ((FY + 2) << lq); e += kPipeThreads) {
                    const int rr = e >> lq, gy = y0 - 1 + rr;
                    if (!row_ok(gy)) continue;
                    const int o = (rr + 1) << lnx;
                    gs_quad<T, CH>(X0 + o, X0 + o - nx, X0 + o + nx, Xm + o, Xp + o, B0 + (rr << lnx), e & qmask, nq,
                                   ((gy & ymask) + gz) & 1, inv, gy, d.ny);
                }
            }
            __syncthreads();
            const int kb = k - 1;
            if (kb >= z0) {
                // black cells of plane k-1 on the tile (z neighbours: k-2 and k)
                const int gz = kb & zmask;
                T* const Ym = xs + (size_t)skm2 * xplane;
                const T* B1 = bs + (size_t)skm1 * bplane;
                for (int e = tid; e < (FY << lq); e += kPipeThreads) {
                    const int rr = e >> lq, gy = y0 + rr;
                    const int o = (rr + 2) << lnx;
                    gs_quad<T, CH>(Xm + o, Xm + o - nx, Xm + o + nx, Ym + o, X0 + o, B1 + ((rr + 1) << lnx), e & qmask,
                                   nq, (gy + gz + 1) & 1, inv, gy, d.ny);
                }
            }
            __syncthreads();
            if (kb >= z0) {
                // plane k-1 of the tile is final
                V* dst = reinterpret_cast<V*>(xout + ((((long long)kb << lny) + y0) << lnx));
                const V* src = reinterpret_cast<const V*>(Xm + 2 * nx);
                for (int e = tid; e < (FY << lq); e += kPipeThreads) dst[e] = src[e];
            }
            // the slot of plane k-2 is free: its last reader, the black update, is behind the barrier
            issue(next, snext);
            ++next;
            snext = next_slot(snext);
            skm1 = sk;
            sk = skp1;
        }
        pipe::wait_pending<0>();
        s_first = (s_first + (next - pfirst)) % R;
        __syncthreads();
    }
}

// Full weighting on 2D (periodic) grids, src/mg/solver.h:153-181: (1,3,3,1)^2/64
// over 16 taps; the 3D form is restrict_cell2.
template <typename T, bool RED>
__device__ __forceinline__ void restrict_cell(const Dims& d, T* coarse, const T* fine, int xc, int yc) {
    int xs[4], ys[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        xs[k] = wrapi(2 * xc - 1 + k, d.nx);
        ys[k] = wrapi(2 * yc - 1 + k, d.ny);
    }
    auto tap = [&](int ky, int kx) { return fine[xs[kx] + d.nx * ys[ky]]; };
    auto row = [&](int ky) { return red_row<T>(ys[ky] & 1, [&](int kx) { return tap(ky, kx); }); };
    coarse[xc + (d.nx / 2) * yc] =
        (RED ? full4<T>(row(0), row(1), row(2), row(3)) : restrict_plane<T>(tap)) * T(1.0 / 64.0);
}

template <typename T, bool RED>
__global__ void k_restrict(Dims d, T* __restrict__ coarse, const T* __restrict__ fine) {
    wait_launch();
    const int xc = blockIdx.x * BX + threadIdx.x, yc = blockIdx.y * BY + threadIdx.y;
    if (xc >= d.nx / 2 || yc >= d.ny / 2) return;
    restrict_cell<T, RED>(d, coarse, fine, xc, yc);
}

// Trilinear prolongation (27,9,3,1)/64, src/mg/solver.h:71-151 (prolong_plane4,
// mg_cells.cuh). One thread per coarse cell writes the eight fine cells between
// it and its +1 neighbours; in channel mode the wall rows take the bilinear
// (9,3,1)/16 weights. C(x, y, z): the coarse values; put(x, y, z, value,
// scale): adds to or sets the fine cell.
template <typename T, bool ADD>
__device__ __forceinline__ void prolong_put(T* fine, long long i, T val, T scale) {
    if (ADD) fine[i] = fma_t(val, scale, fine[i]);
    else fine[i] = val * scale;
}
// BLACK: on the black cells only (prolong_before_sweep)
template <typename T, bool BLACK, typename C, typename P>
__device__ __forceinline__ void prolong_cell_any(const Dims& d, int xc, int yc, int zc, int xn, int yn, int zn,
                                                 const int (&xf)[2], const int (&yf)[2], const int (&zf)[2], C cv,
                                                 P put) {
    const int cy = d.ny / 2;
    if (!d.channel || yc < cy - 1) {
        const T blb = cv(xc, yc, zc), brb = cv(xn, yc, zc), ulb = cv(xc, yn, zc), urb = cv(xn, yn, zc);
        const T blf = cv(xc, yc, zn), brf = cv(xn, yc, zn), ulf = cv(xc, yn, zn), urf = cv(xn, yn, zn);
        prolong_plane4(blb, brb, ulb, urb, blf, brf, ulf, urf, BLACK, 0,
                       [&](int rx, int ry, T v, T s) { put(xf[rx], yf[ry], zf[0], v, s); });
        prolong_plane4(blf, brf, ulf, urf, blb, brb, ulb, urb, BLACK, 1,
                       [&](int rx, int ry, T v, T s) { put(xf[rx], yf[ry], zf[1], v, s); });
    }
    if (d.channel && (yc == 0 || yc == cy - 1)) {
        for (int side = 0; side < 2; ++side) {  // a thread with cy == 1 owns both wall rows
            if (side == 0 && yc != 0) continue;
            if (side == 1 && yc != cy - 1) continue;
            const int yw = side == 0 ? 0 : d.ny - 1, ry = 1 - side;  // row 0 is even, ny - 1 odd
            const T bl = cv(xc, yc, zc), br = cv(xn, yc, zc), fl = cv(xc, yc, zn), fr = cv(xn, yc, zn);
            prolong_row2(bl, br, fl, fr, black_col(BLACK, ry, 0), [&](int rx, T v, T s) { put(xf[rx], yw, zf[0], v, s); });
            prolong_row2(fl, fr, bl, br, black_col(BLACK, ry, 1), [&](int rx, T v, T s) { put(xf[rx], yw, zf[1], v, s); });
        }
    }
}
// 2D (periodic) grids: bilinear (9,3,3,1)/16 onto the four fine cells
template <typename T, bool ADD, bool BLACK>
__device__ __forceinline__ void prolong_cell(const Dims& d, T* fine, const T* coarse, int xc, int yc) {
    const int cx = d.nx / 2, cy = d.ny / 2;
    const int xn = xc + 1 == cx ? 0 : xc + 1, yn = yc + 1 == cy ? 0 : yc + 1;
    const int xf[2] = {2 * xc + 1, (2 * xc + 2) % d.nx}, yf[2] = {2 * yc + 1, (2 * yc + 2) % d.ny};
    auto C2 = [&](int a, int b) { return coarse[a + cx * b]; };
    const T bl = C2(xc, yc), br = C2(xn, yc), ul = C2(xc, yn), ur = C2(xn, yn);
    prolong_row2(bl, br, ul, ur, black_col(BLACK, 0, 1),
                 [&](int rx, T v, T s) { prolong_put<T, ADD>(fine, xf[rx] + d.nx * yf[0], v, s); });
    prolong_row2(ul, ur, bl, br, black_col(BLACK, 1, 1),
                 [&](int rx, T v, T s) { prolong_put<T, ADD>(fine, xf[rx] + d.nx * yf[1], v, s); });
}

// 3D levels with Ix2 or IxG indexing. Restriction: 64 taps (1,3,3,1)^3/512 around
// the coarse cell (restrict_taps, mg_cells.cuh); y clamps at the channel walls,
// wraps in periodic mode.
template <typename T, bool RED, typename IX>
__device__ __forceinline__ void restrict_cell2(const Dims& d, const IX& I, T* coarse, const T* fine, int xc, int yc,
                                               int zc) {
    int xs[4], ys[4], zs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = 2 * xc - 1 + k, y = 2 * yc - 1 + k;
        xs[k] = k == 0 ? I.xm(2 * xc) : (k == 3 ? I.xp(2 * xc + 1) : x);
        zs[k] = I.wz(2 * zc - 1 + k);
        if (d.channel) ys[k] = y < 0 ? 0 : (y > d.ny - 1 ? d.ny - 1 : y);
        else ys[k] = k == 0 ? I.ym(2 * yc) : (k == 3 ? I.yp(2 * yc + 1) : y);
    }
    const int o = I.coarse(xc, yc, zc);
    if (RED)
        coarse[o] = restrict_rows<T>([&](int kz, int ky) {
            // the row's y comes clamped at channel walls
            return red_row<T>(((ys[ky] + zs[kz]) & 1) != 0, [&](int kx) { return fine[I.at(xs[kx], ys[ky], zs[kz])]; });
        });
    else
        coarse[o] = restrict_taps<T>([&](int kz, int ky, int kx) { return fine[I.at(xs[kx], ys[ky], zs[kz])]; });
}

template <typename T, bool RED, typename IX>
__global__ void k_restrict2(Dims d, T* __restrict__ coarse, const T* __restrict__ fine, int rev) {
    wait_launch();
    const IX I(d);
    const uint3 B = block_at(rev);
    const int xc = B.x * BX + threadIdx.x, yc = B.y * BY + threadIdx.y, zc = B.z;
    if (xc >= d.nx / 2 || yc >= d.ny / 2) return;
    restrict_cell2<T, RED>(d, I, coarse, fine, xc, yc, zc);
}

template <typename T, bool ADD, bool BLACK, typename IX>
__device__ __forceinline__ void prolong_cell2(const Dims& d, const IX& I, T* fine, const T* coarse, int xc, int yc,
                                              int zc) {
    const int cx = d.nx / 2, cy = d.ny / 2, cz = d.nz / 2;
    const int xf[2] = {2 * xc + 1, I.xp(2 * xc + 1)}, yf[2] = {2 * yc + 1, I.yp(2 * yc + 1)},
              zf[2] = {2 * zc + 1, I.zp(2 * zc + 1)};
    prolong_cell_any<T, BLACK>(
        d, xc, yc, zc, xc + 1 == cx ? 0 : xc + 1, yc + 1 == cy ? 0 : yc + 1, zc + 1 == cz ? 0 : zc + 1, xf, yf, zf,
        [&](int a, int b, int c) { return coarse[I.coarse(a, b, c)]; },
        [&](int a, int b, int c, T v, T s) { prolong_put<T, ADD>(fine, I.at(a, b, c), v, s); });
}

// Fine-level residual fused with the full-weighting restriction. A block takes RR_T x RR_T coarse columns
// and RR_CZ coarse planes; r = b - L x of its fine tile (2 RR_T + 2 cells a
// side: the taps reach one fine cell beyond the tile's own) is formed in
// shared memory, one fine plane at a time, in a ring of the four planes the
// current coarse plane reads, and every coarse cell sums its 64 taps from the
// ring. The residual is k_residual_z2's expression and the sum is
// restrict_cell2's, so the coarse right-hand side equals the two
// kernels' bit for bit, and the fine residual is never written to memory.
constexpr int RR_T = 16, RR_F = 2 * RR_T + 2, RR_THREADS = RR_T * RR_T;
// ring plane layout: row stride RR_RS, even columns first and odd columns
// from RR_ODD, so that the 16 coarse cells of a half warp read 16
// consecutive words and the two halves (two fine rows apart) the other 16
// banks: no shared-memory bank conflicts in the tap loop
constexpr int RR_RS = 40, RR_ODD = 20;
__device__ __forceinline__ int rr_at(int jy, int jx) { return jy * RR_RS + (jx & 1) * RR_ODD + (jx >> 1); }

template <typename T, int RR_CZ>
__global__ void __launch_bounds__(RR_THREADS) k_resid_restrict2(Dims d, T* __restrict__ cb,
                                                               const T* __restrict__ xv, const T* __restrict__ b,
                                                               int rev, bool red) {
    wait_launch();
    __shared__ T ring[4][RR_F * RR_RS];
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int xc0 = B.x * RR_T, yc0 = B.y * RR_T, zc0 = B.z * RR_CZ;
    const int xf0 = 2 * xc0 - 1, yf0 = 2 * yc0 - 1;  // fine cell of tile column / row 0 (unwrapped)
    const T off = T(d.n) * T(d.n);
    const int tid = threadIdx.x;
    // residual of fine plane zf (unwrapped) into its ring slot; channel rows
    // beyond the walls are never tapped (the taps clamp) and stay unset
    auto fill = [&](int zf) {
        T* dst = ring[zf & 3];
        const int z = zf & I.mz;
        for (int e = tid; e < RR_F * RR_F; e += RR_THREADS) {
            const int jy = e / RR_F, jx = e - jy * RR_F;
            int y = yf0 + jy;
            if (d.channel) {
                if (y < 0 || y >= d.ny) continue;
            } else {
                y &= I.my;
            }
            const int x = (xf0 + jx) & I.mx;
            if (red && ((x + y + z) & 1)) {  // restrict_after_sweep
                dst[rr_at(jy, jx)] = T(0);
                continue;
            }
            T S;
            int c;
            lap_row2(d, I, xv, x, y, z, S, c);
            const int i = I.at(x, y, z);
            dst[rr_at(jy, jx)] = b[i] - off * (S - lap_count<T>(c) * xv[i]);
        }
    };
    const int cxl = tid % RR_T, cyl = tid / RR_T;
    const int xc = xc0 + cxl, yc = yc0 + cyl;
    int col[4], row[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int dd = k - 2;
        col[k] = (k & 1) * RR_ODD + cxl + (k >> 1);  // tile column 2 cxl + k: fine x = 2 xc + 1 + dd
        int yy;
        if (d.channel) {
            const int ycf = 2 * yc + 1;
            yy = ycf + (dd > -ycf ? dd : -ycf);
            yy = yy < d.ny - 1 ? yy : d.ny - 1;
        } else {
            yy = 2 * yc + 1 + dd;  // unwrapped: the ring holds the wrapped values in order
        }
        row[k] = yy - yf0;
    }
    fill(2 * zc0 - 1);
    fill(2 * zc0);
    for (int zc = zc0; zc < zc0 + RR_CZ; ++zc) {
        fill(2 * zc + 1);
        fill(2 * zc + 2);
        __syncthreads();
        const T acc = restrict_taps<T>(
            [&](int kz, int ky, int kx) { return ring[(2 * zc - 1 + kz) & 3][row[ky] * RR_RS + col[kx]]; });
        const int o = xc | (yc << (I.lx - 1)) | (zc << (I.lxy - 2));
        cb[o] = acc;
        __syncthreads();  // the next fills overwrite the two oldest planes
    }
}

template <typename T, bool ADD, bool BLACK, typename IX>
__global__ void k_prolong2(Dims d, T* __restrict__ fine, const T* __restrict__ coarse, int rev) {
    wait_launch();
    const IX I(d);
    const uint3 B = block_at(rev);
    const int xc = B.x * BX + threadIdx.x, yc = B.y * BY + threadIdx.y, zc = B.z;
    if (xc >= d.nx / 2 || yc >= d.ny / 2) return;
    prolong_cell2<T, ADD, BLACK>(d, I, fine, coarse, xc, yc, zc);
}

template <typename T, bool ADD, bool BLACK>
__global__ void k_prolong(Dims d, T* __restrict__ fine, const T* __restrict__ coarse) {
    wait_launch();
    const int xc = blockIdx.x * BX + threadIdx.x, yc = blockIdx.y * BY + threadIdx.y;
    if (xc >= d.nx / 2 || yc >= d.ny / 2) return;
    prolong_cell<T, ADD, BLACK>(d, fine, coarse, xc, yc);
}

// Column-marching transfers for 3D power-of-two levels whose coarse x extent
// is a multiple of 32 and coarse y extent a multiple of kTrBY. A warp holds 32
// consecutive coarse x of one coarse row, so its fine accesses are the 64
// consecutive cells 2 xc .. 2 xc + 63 of a fine row, read or written as one
// pair per lane (256 contiguous bytes for FP32); the cells one beyond a lane's
// pair come from the adjacent lane by a shuffle (the first and last lanes load
// them). A thread then walks CZ coarse planes along z. The one-cell kernels
// (restrict_cell2, prolong_cell2) read and write with a stride of two cells,
// 64 single loads per coarse cell in the restriction, and their prolongation
// stores wait on the loads of the next cell (same array): on 256^3 both ran at
// a third of the copy bandwidth.
constexpr int kTrBY = 8;
template <typename T>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};

// Full weighting with restrict_cell2's arithmetic (restrict_plane, full4):
// fine planes 2 zc + 1 and 2 zc + 2 are the last two planes of coarse plane zc
// and the first two of zc + 1, so each fine plane is read and summed once and
// its sum serves two coarse planes: the same bits with half the sums.
//
// A lane reads 16 bytes of each fine tap row (CE = 4 FP32 or 2 FP64 cells)
// and takes the cells on either side from its neighbours, so it serves CE / 2
// coarse cells: a warp covers 16 CE coarse x. The block's fine tile of a plane
// (rows 2 yc0 - 1 .. 2 yc0 + 16, clamped at channel walls, wrapped otherwise;
// 32 CE cells from 2 xc0 and one 16-byte chunk on either side, wrapped in x)
// arrives in shared memory by 16-byte asynchronous copies issued
// kTrStages - 1 planes ahead, one commit group per plane, so that the march
// along z keeps two planes of DRAM reads in flight with one barrier per plane.
constexpr int kTrStages = 3;
constexpr int kTrRows = 2 * kTrBY + 2;
template <typename T>
struct TrTile {
    static constexpr int CE = 16 / (int)sizeof(T);       // cells per 16-byte chunk (per lane)
    static constexpr int CX = 16 * CE;                    // coarse x per block
    static constexpr int W = 34 * CE;                     // row: left chunk, 32 lane chunks, right chunk
    static constexpr int CHUNKS = kTrRows * 34;           // 16-byte chunks per plane
    static constexpr int PER_THREAD = (CHUNKS + 32 * kTrBY - 1) / (32 * kTrBY);
};
template <typename T>
struct Quad;
template <>
struct Quad<float> {
    using type = float4;
};
template <>
struct Quad<double> {
    using type = double2;
};
template <typename T>
__device__ __forceinline__ void quad_get(const T* p, T (&v)[16 / sizeof(T)]) {
    const typename Quad<T>::type q = *reinterpret_cast<const typename Quad<T>::type*>(p);
    if constexpr (sizeof(T) == 4) {
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        v[0] = q.x; v[1] = q.y;
    }
}

template <typename T, int CZ>
__global__ void __launch_bounds__(32 * kTrBY) k_restrict_cols(Dims d, T* __restrict__ coarse,
                                                              const T* __restrict__ fine, int rev) {
    wait_launch();
    using TT = TrTile<T>;
    constexpr int CE = TT::CE, M = CE / 2;  // M coarse cells per lane
    constexpr int NP = 2 * CZ + 2;          // fine planes of the block
    __shared__ __align__(16) T st[kTrStages][kTrRows * TT::W];
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int lane = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + lane;
    const int xc0 = B.x * TT::CX, yc0 = B.y * kTrBY, zc0 = B.z * CZ;
    // this thread's chunks of every plane: source offset within the plane
    // (-1: none) and destination offset within the stage
    int src[TT::PER_THREAD], dst[TT::PER_THREAD];
#pragma unroll
    for (int u = 0; u < TT::PER_THREAD; ++u) {
        const int c = tid + u * 32 * kTrBY;
        src[u] = -1;
        dst[u] = 0;
        if (c < TT::CHUNKS) {
            const int j = c / 34, k = c - j * 34;
            int y = 2 * yc0 - 1 + j;
            if (d.channel) y = y < 0 ? 0 : (y > d.ny - 1 ? d.ny - 1 : y);
            else y &= I.my;
            src[u] = ((2 * xc0 - CE + k * CE) & I.mx) | (y << I.lx);
            dst[u] = j * TT::W + k * CE;
        }
    }
    // copies of fine plane 2 zc0 - 1 + i; a commit group per plane, empty
    // past the block's last plane, so that the group count is the plane count
    auto issue = [&](int i) {
        if (i < NP) {
            T* stage = st[i % kTrStages];
            const T* pl = fine + (((2 * zc0 - 1 + i) & I.mz) << I.lxy);
#pragma unroll
            for (int u = 0; u < TT::PER_THREAD; ++u)
                if (src[u] >= 0) pipe::cp16(stage + dst[u], pl + src[u]);
        }
        pipe::commit();
    };
    auto acquire = [&](int i) -> const T* {
        pipe::wait_pending<kTrStages - 2>();
        __syncthreads();           // plane i is in; plane i - 1 is read by every thread
        issue(i + kTrStages - 1);  // into plane i - 1's stage
        return st[i % kTrStages];
    };
    // the taps of a staged plane: e[ky][1 + q] = fine x = 2 xc0 + CE lane + q,
    // q = -1 .. CE (rows 2 ty + ky of the tile)
    auto taps = [&](const T* pl, T (&e)[4][CE + 2]) {
#pragma unroll
        for (int ky = 0; ky < 4; ++ky) {
            const T* row = pl + (2 * ty + ky) * TT::W + CE;  // fine x = 2 xc0
            T v[CE];
            quad_get(row + CE * lane, v);
            T l = __shfl_up_sync(0xffffffffu, v[CE - 1], 1), r = __shfl_down_sync(0xffffffffu, v[0], 1);
            if (lane == 0) l = row[-1];
            if (lane == 31) r = row[32 * CE];
            e[ky][0] = l;
#pragma unroll
            for (int q = 0; q < CE; ++q) e[ky][1 + q] = v[q];
            e[ky][CE + 1] = r;
        }
    };
    // a plane's sum for coarse cell m of the lane: taps fine x = 2 xc - 1 ..
    // 2 xc + 2 = e[ky][2m .. 2m + 3]
    auto plane = [&](T (&p)[M], const T (&e)[4][CE + 2]) {
#pragma unroll
        for (int m = 0; m < M; ++m) p[m] = restrict_plane<T>([&](int ky, int kx) { return e[ky][2 * m + kx]; });
    };
#pragma unroll
    for (int i = 0; i < kTrStages - 1; ++i) issue(i);
    T p0[M], p1[M], p2[M], p3[M], e[4][CE + 2];
    taps(acquire(0), e);
    plane(p0, e);
    taps(acquire(1), e);
    plane(p1, e);
    const int co = (xc0 + M * lane) | ((yc0 + ty) << (I.lx - 1));
    for (int k = 0; k < CZ; ++k) {
        taps(acquire(2 * k + 2), e);
        plane(p2, e);
        taps(acquire(2 * k + 3), e);
        plane(p3, e);
        T acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = full4<T>(p0[m], p1[m], p2[m], p3[m]) * T(1.0 / 512.0);
        const int o = co | ((zc0 + k) << (I.lxy - 2));
        if constexpr (M == 2) {
            *reinterpret_cast<float2*>(coarse + o) = make_float2(acc[0], acc[1]);
        } else {
            coarse[o] = acc[0];
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            p0[m] = p2[m];
            p1[m] = p3[m];
        }
    }
    pipe::wait_pending<0>();
}

// FP32 fine-level residual fused with the column restriction: the block of
// k_restrict_cols (64 coarse x, kTrBY coarse y, CZ coarse planes) forms the
// residual r = b - L x of each fine plane of its tile in shared memory and
// restricts from there, so the fine residual never goes to memory. x planes
// (rows 2 yc0 - 2 .. 2 yc0 + 17, 36 16-byte chunks a row from x = 2 xc0 - 8)
// and b planes (rows 2 yc0 - 1 .. 2 yc0 + 16, 34 chunks from 2 xc0 - 4)
// arrive by asynchronous copies issued two planes ahead into rings of kRrX
// and kRrB slots; per fine plane there are two barriers (the plane's inputs
// are in and the previous taps are done / the residual plane is written).
// The residual plane holds 34 chunks a row (x = 2 xc0 - 4 .. 2 xc0 + 131, the
// layout k_restrict_cols stages): each thread forms whole chunks, four cells
// from 16-byte words and the cells on either side by single loads. Every
// residual is k_residual_z2's expression in its order and the sums are
// k_restrict_cols', so the coarse right-hand side
// equals the two kernels' bit for bit. In channel mode the rows beyond the
// walls take the residual of the wall row, as the restriction's clamped taps
// read it.
constexpr int kRrX = 4, kRrB = 4, kRrXRows = 2 * kTrBY + 4;
constexpr int kRrXW = 144, kRrW = 136;  // floats a staged x row (36 chunks) / b and residual row (34)
constexpr int kRrTasks = kTrRows * 34;  // residual chunks a plane
constexpr int kRrPT = (kRrTasks + 32 * kTrBY - 1) / (32 * kTrBY);
// Split rows (Split2) are staged as 72 even cells, then 72 odd ones, from x = 2 xc0 - 8
// for x and for b (a colour's half of a row goes to one of the two by the parity of
// y + z), and read from there by pairs.
constexpr int kRrBW = 144, kRrHalf = 72;
constexpr size_t kRrSmem = sizeof(float) * ((size_t)kRrX * kRrXRows * kRrXW + (size_t)kRrB * kTrRows * kRrBW +
                                            (size_t)kTrRows * kRrW);

template <int CZ, bool CH, bool SPLIT>
__global__ void __launch_bounds__(32 * kTrBY, 2) k_resid_restrict_cols(Dims d, float* __restrict__ cb,
                                                                    const float* __restrict__ xv,
                                                                    const float* __restrict__ bv, int rev) {
    wait_launch();
    constexpr int NP = 2 * CZ + 2;  // fine planes restricted (residuals formed)
    constexpr int NI = NP + 2;      // staged items: x planes 2 zc0 - 2 .. 2 zc0 + 2 CZ + 1
    constexpr int XCH = (kRrXRows * 36 + 32 * kTrBY - 1) / (32 * kTrBY);
    constexpr int BC = SPLIT ? 36 : 34, BW = SPLIT ? kRrBW : kRrW;  // chunks and floats a staged b row
    constexpr int BCH = (kTrRows * BC + 32 * kTrBY - 1) / (32 * kTrBY);
    extern __shared__ __align__(16) float rr_smem[];
    float* xs = rr_smem;                          // [kRrX][kRrXRows][kRrXW]
    float* bs = xs + kRrX * kRrXRows * kRrXW;     // [kRrB][kTrRows][BW]
    float* rs = bs + kRrB * kTrRows * BW;         // [kTrRows][kRrW]
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int lane = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + lane;
    const int xc0 = B.x * 64, yc0 = B.y * kTrBY, zc0 = B.z * CZ;
    auto yrow = [&](int y) {  // a row in range: clamped at channel walls, wrapped otherwise
        if (CH) return y < 0 ? 0 : (y > d.ny - 1 ? d.ny - 1 : y);
        return y & I.my;
    };
    // this thread's chunks of every x / b plane: source offset within the
    // plane (-1: none), destination offset within the slot
    int xsrc[XCH], xdst[XCH], bsrc[BCH], bdst[BCH];
    // split rows: chunk k of row y holds four cells of colour k / 18; on a plane of
    // parity 0 they go to the half h = (y + k / 18) & 1, on the others to 1 - h (bit 0
    // of the destination, the offsets being multiples of four)
    auto chunk = [&](int k, int y, int& src, int& dst) {
        const int h = k / 18, kk = k - 18 * h;
        src = ((xc0 - 4 + 4 * kk) & (I.mx >> 1)) | (h << (I.lx - 1)) | (y << I.lx);
        dst = (4 * kk) | ((y + h) & 1);
    };
    auto to = [&](int dst, int k) { return SPLIT ? (dst & ~1) + kRrHalf * ((dst + k) & 1) : dst; };
#pragma unroll
    for (int u = 0; u < XCH; ++u) {
        const int c = tid + u * 32 * kTrBY;
        xsrc[u] = -1;
        xdst[u] = 0;
        if (c < kRrXRows * 36) {
            const int j = c / 36, k = c - j * 36;
            if (SPLIT) {
                chunk(k, yrow(2 * yc0 - 2 + j), xsrc[u], xdst[u]);
                xdst[u] += j * kRrXW;
            } else {
                xsrc[u] = ((2 * xc0 - 8 + 4 * k) & I.mx) | (yrow(2 * yc0 - 2 + j) << I.lx);
                xdst[u] = j * kRrXW + 4 * k;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < BCH; ++u) {
        const int c = tid + u * 32 * kTrBY;
        bsrc[u] = -1;
        bdst[u] = 0;
        if (c < kTrRows * BC) {
            const int j = c / BC, k = c - j * BC;
            if (SPLIT) {
                chunk(k, yrow(2 * yc0 - 1 + j), bsrc[u], bdst[u]);
                bdst[u] += j * BW;
            } else {
                bsrc[u] = ((2 * xc0 - 4 + 4 * k) & I.mx) | (yrow(2 * yc0 - 1 + j) << I.lx);
                bdst[u] = j * BW + 4 * k;
            }
        }
    }
    // this thread's residual chunks: residual row jr, chunk k (cells
    // x = 2 xc0 - 4 + 4 k ..); the x-tile row of the residual's row (channel:
    // the wall row for the rows beyond it) and its wall flags
    int tr[kRrPT], tx[kRrPT], tb[kRrPT];
    bool tym[kRrPT], typ[kRrPT];
#pragma unroll
    for (int u = 0; u < kRrPT; ++u) {
        const int t = tid + u * 32 * kTrBY;
        tr[u] = -1;
        tx[u] = 0;
        tb[u] = 0;
        tym[u] = typ[u] = true;
        if (t < kRrTasks) {
            const int jr = t / 34, k = t - jr * 34;
            const int y = 2 * yc0 - 1 + jr;
            const int ye = CH ? (y < 0 ? 0 : (y > d.ny - 1 ? d.ny - 1 : y)) : y;
            const int jx = ye - (2 * yc0 - 2);
            tr[u] = jr * kRrW + 4 * k;
            tb[u] = jr * BW + (SPLIT ? 2 * k + 2 : 4 * k);
            tx[u] = jx * kRrXW + (SPLIT ? 2 * k + 2 : 4 * k + 4);
            tym[u] = !CH || ye > 0;
            typ[u] = !CH || ye < d.ny - 1;
        }
    }
    // item k: x plane 2 zc0 - 2 + k, and b of the same plane for 1 <= k <= NP;
    // one commit group per item, empty past the last
    auto issue = [&](int k) {
        if (k < NI) {
            const int zo = ((2 * zc0 - 2 + k) & I.mz) << I.lxy;
            float* xd = xs + (k % kRrX) * kRrXRows * kRrXW;
            const float* xsp = xv + zo;
#pragma unroll
            for (int u = 0; u < XCH; ++u)
                if (xsrc[u] >= 0) pipe::cp16(xd + to(xdst[u], k), xsp + xsrc[u]);
            if (k >= 1 && k <= NP) {
                float* bd = bs + (k % kRrB) * kTrRows * BW;
                const float* bsp = bv + zo;
#pragma unroll
                for (int u = 0; u < BCH; ++u)
                    if (bsrc[u] >= 0) pipe::cp16(bd + to(bdst[u], k), bsp + bsrc[u]);
            }
        }
        pipe::commit();
    };
    const float off = float(d.n) * float(d.n);
    auto cell = [&](float x0, float xl, float xr, float zm, float zp, float ym, float yp, float b, bool hm, bool hp) {
        float S = (xl + xr) + (zm + zp);
        float c = 6.f;
        if (CH) {
            if (hm) S += ym; else c -= 1.f;
            if (hp) S += yp; else c -= 1.f;
        } else {
            S += ym + yp;
        }
        return b - off * (S - c * x0);
    };
    // residual chunks of fine plane i (fine z = 2 zc0 - 1 + i) into rs
    auto resid = [&](int i) {
        const float* xc = xs + ((i + 1) % kRrX) * kRrXRows * kRrXW;
        const float* xm = xs + (i % kRrX) * kRrXRows * kRrXW;        // z - 1
        const float* xp = xs + ((i + 2) % kRrX) * kRrXRows * kRrXW;  // z + 1
        const float* bp = bs + ((i + 1) % kRrB) * kTrRows * BW;
        // four cells from x = 2 xc0 - 4 + 4 k
        auto four = [](const float* p) {
            if (!SPLIT) return *reinterpret_cast<const float4*>(p);
            const float2 e = *reinterpret_cast<const float2*>(p), o = *reinterpret_cast<const float2*>(p + kRrHalf);
            return make_float4(e.x, o.x, e.y, o.y);
        };
#pragma unroll
        for (int u = 0; u < kRrPT; ++u) {
            if (tr[u] < 0) break;
            const float* c0 = xc + tx[u];
            const float4 v = four(c0);
            const float4 vym = four(c0 - kRrXW);
            const float4 vyp = four(c0 + kRrXW);
            const float4 vzm = four(xm + tx[u]);
            const float4 vzp = four(xp + tx[u]);
            const float4 vb = four(bp + tb[u]);
            const float l = SPLIT ? c0[kRrHalf - 1] : c0[-1], r = SPLIT ? c0[2] : c0[4];
            const bool hm = tym[u], hp = typ[u];
            float4 o;
            o.x = cell(v.x, l, v.y, vzm.x, vzp.x, vym.x, vyp.x, vb.x, hm, hp);
            o.y = cell(v.y, v.x, v.z, vzm.y, vzp.y, vym.y, vyp.y, vb.y, hm, hp);
            o.z = cell(v.z, v.y, v.w, vzm.z, vzp.z, vym.z, vyp.z, vb.z, hm, hp);
            o.w = cell(v.w, v.z, r, vzm.w, vzp.w, vym.w, vyp.w, vb.w, hm, hp);
            *reinterpret_cast<float4*>(rs + tr[u]) = o;
        }
    };
    // the restriction taps of the residual plane for this thread: e[ky][1 + q]
    // = fine x = 2 xc0 + 4 lane + q, q = -1 .. 4 (k_restrict_cols' taps)
    auto taps = [&](float (&e)[4][6]) {
#pragma unroll
        for (int ky = 0; ky < 4; ++ky) {
            const float* row = rs + (2 * ty + ky) * kRrW + 4;  // fine x = 2 xc0
            const float4 q = *reinterpret_cast<const float4*>(row + 4 * lane);
            float l = __shfl_up_sync(0xffffffffu, q.w, 1), r = __shfl_down_sync(0xffffffffu, q.x, 1);
            if (lane == 0) l = row[-1];
            if (lane == 31) r = row[128];
            e[ky][0] = l;
            e[ky][1] = q.x;
            e[ky][2] = q.y;
            e[ky][3] = q.z;
            e[ky][4] = q.w;
            e[ky][5] = r;
        }
    };
    // the last four planes' sums, oldest first
    float p[4][2], e[4][6];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k][0] = p[k][1] = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) issue(k);
    const int co = (xc0 + 2 * lane) | ((yc0 + ty) << (I.lx - 1));
    for (int i = 0; i < NP; ++i) {
        pipe::wait_pending<1>();  // items <= i + 2 are in
        __syncthreads();          // ... for every thread; the last plane's taps are done
        resid(i);
        __syncthreads();          // the residual plane is written; x item i and b item i + 1 are free
        issue(i + 4);
        taps(e);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            p[0][m] = p[1][m];
            p[1][m] = p[2][m];
            p[2][m] = p[3][m];
            p[3][m] = restrict_plane<float>([&](int ky, int kx) { return e[ky][2 * m + kx]; });
        }
        if (i >= 3 && (i & 1)) {
            const int o = co | ((zc0 + (i - 3) / 2) << (I.lxy - 2));
            const float a0 = full4<float>(p[0][0], p[1][0], p[2][0], p[3][0]) * float(1.0 / 512.0);
            const float a1 = full4<float>(p[0][1], p[1][1], p[2][1], p[3][1]) * float(1.0 / 512.0);
            *reinterpret_cast<float2*>(cb + o) = make_float2(a0, a1);
        }
    }
    pipe::wait_pending<0>();
}

// Trilinear prolongation-add with prolong_cell2's arithmetic. A thread owns
// the fine pairs x = 2t, 2t+1 of rows y = 2s, 2s+1 in planes z = 2r, 2r+1, all
// eight nearest to coarse cell (t, s, r): fine cell 2t + 1 is the first (xcf)
// of coarse cell t and 2t the second (xnf) of coarse cell t - 1, and likewise
// in y and z, so they need the coarse values at t - 1 .. t + 1, s - 1 .. s + 1,
// r - 1 .. r + 1, kept in registers as a window of three coarse planes that
// moves one plane per r. The sums run along z, then y, then x as in
// prolong_plane4 and share their partial sums, and in channel mode the wall
// rows y = 0 and ny - 1 take the wall expressions: the same bits. The block's
// fine values of plane pair r (2 x 16 rows of 64 cells) and its tile of
// coarse plane r + 1 arrive in shared memory by 16-byte asynchronous copies
// issued one or two plane pairs ahead (FP64 / FP32); the sums go straight to
// memory.
template <typename T>
struct ProTile {
    static constexpr int CE = 16 / (int)sizeof(T);
    static constexpr int S = sizeof(T) == 4 ? 3 : 2;   // stages (static shared memory <= 48 KB)
    static constexpr int FROWS = 4 * kTrBY;            // 2 planes x 2 kTrBY rows
    static constexpr int FW = 64;
    static constexpr int CROWS = kTrBY + 2;
    static constexpr int CW = 32 + 2 * CE;
    static constexpr int STAGE = FROWS * FW + CROWS * CW;
};

template <typename T, int RZ, bool SPLIT>
__global__ void __launch_bounds__(32 * kTrBY) k_prolong_cols(Dims d, T* __restrict__ fine,
                                                             const T* __restrict__ coarse, int rev) {
    wait_launch();
    using P2 = typename Pair<T>::type;
    using PT = ProTile<T>;
    constexpr int CE = PT::CE;
    __shared__ __align__(16) T st[PT::S][PT::STAGE];
    const Ix2 I(d);
    const uint3 B = block_at(rev);
    const int lane = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + lane;
    const int cx = d.nx / 2, cy = d.ny / 2, cz = d.nz / 2, lcx = I.lx - 1, lcxy = I.lxy - 2;
    const int t0 = B.x * 32, s0 = B.y * kTrBY, r0 = B.z * RZ;
    const int t = t0 + lane, s = s0 + ty;
    auto crow = [&](int y) {  // coarse row y in range: clamped at channel walls, wrapped otherwise
        if (d.channel) return y < 0 ? 0 : (y > cy - 1 ? cy - 1 : y);
        return y & (cy - 1);
    };
    // item i: the fine values of plane pair r0 + i and the coarse tile of
    // plane r0 + i + 1; a commit group per item, empty past the last
    auto issue = [&](int i) {
        if (i < RZ) {
            T* dst = st[i % PT::S];
            const int r = r0 + i;
            for (int c = tid; c < PT::FROWS * (PT::FW / CE); c += 32 * kTrBY) {
                const int j = c / (PT::FW / CE), k = c - j * (PT::FW / CE);
                const int jz = j / (2 * kTrBY), jy = j - jz * (2 * kTrBY);
                const int row = ((2 * s0 + jy) << I.lx) | ((2 * r + jz) << I.lxy);
                if (SPLIT) {  // staged as 32 even cells, then 32 odd ones
                    constexpr int HC = PT::FW / CE / 2;
                    const int h = k / HC, kk = k - h * HC;
                    pipe::cp16(dst + j * PT::FW + ((jy + jz + h) & 1) * 32 + kk * CE,
                               fine + ((t0 + kk * CE) | (h << (I.lx - 1)) | row));
                } else {
                    pipe::cp16(dst + j * PT::FW + k * CE, fine + ((2 * t0 + k * CE) | row));
                }
            }
            T* cdst = dst + PT::FROWS * PT::FW;
            const T* cpl = coarse + (((r + 1) & (cz - 1)) << lcxy);
            for (int c = tid; c < PT::CROWS * (PT::CW / CE); c += 32 * kTrBY) {
                const int j = c / (PT::CW / CE), k = c - j * (PT::CW / CE);
                const int x = (t0 - CE + k * CE) & (cx - 1);
                pipe::cp16(cdst + j * PT::CW + k * CE, cpl + (x | (crow(s0 - 1 + j) << lcx)));
            }
        }
        pipe::commit();
    };
    auto acquire = [&](int i) -> const T* {
        pipe::wait_pending<PT::S - 2>();
        __syncthreads();           // item i is in; item i - 1 is read by every thread
        issue(i + PT::S - 1);      // into item i - 1's stage
        return st[i % PT::S];
    };
#pragma unroll
    for (int i = 0; i < PT::S - 1; ++i) issue(i);
    const bool wall_lo = d.channel && s == 0, wall_hi = d.channel && s == cy - 1;
    // window: coarse planes r - 1, r, r + 1 at rows s - 1 .. s + 1, cells t - 1 .. t + 1
    T w[3][3][3];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                w[p][j][i] = coarse[((t - 1 + i) & (cx - 1)) | (crow(s - 1 + j) << lcx) |
                                    (((r0 - 1 + p) & (cz - 1)) << lcxy)];
    for (int k = 0; k < RZ; ++k) {
        const int r = r0 + k;
        const T* sf = acquire(k);
        const T* sc = sf + PT::FROWS * PT::FW;
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) w[2][j][i] = sc[(ty + j) * PT::CW + CE + lane - 1 + i];
#pragma unroll
        for (int jz = 0; jz < 2; ++jz) {
            // fine plane 2r + jz: near coarse plane r, far r - 1 or r + 1 (z, then y, then x)
            T q[3][3];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int i = 0; i < 3; ++i) q[j][i] = near4(w[1][j][i], w[2 * jz][j][i]);
#pragma unroll
            for (int jy = 0; jy < 2; ++jy) {
                const bool wl = jy == 0 ? wall_lo : wall_hi;  // a wall row has no y neighbour
                T h[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) h[i] = wl ? q[1][i] : near4(q[1][i], q[2 * jy][i]);
                const T sc1 = wl ? T(1.0 / 16.0) : T(1.0 / 64.0);
                // fine x = 2t (nearest to t, far t - 1), 2t + 1 (far t + 1)
                const T* sr = sf + (jz * 2 * kTrBY + 2 * ty + jy) * PT::FW;
                P2 old, out;
                if (SPLIT) {
                    old.x = sr[lane];
                    old.y = sr[32 + lane];
                } else {
                    old = *reinterpret_cast<const P2*>(sr + 2 * lane);
                }
                out.x = fma_t(near4(h[1], h[0]), sc1, old.x);
                out.y = fma_t(near4(h[1], h[2]), sc1, old.y);
                const int row = ((2 * s + jy) << I.lx) | ((2 * r + jz) << I.lxy), p = (jy + jz) & 1;
                if (SPLIT) {
                    fine[t | (p << (I.lx - 1)) | row] = out.x;
                    fine[t | ((1 - p) << (I.lx - 1)) | row] = out.y;
                } else {
                    *reinterpret_cast<P2*>(fine + ((2 * t) | row)) = out;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                w[0][j][i] = w[1][j][i];
                w[1][j][i] = w[2][j][i];
            }
    }
    pipe::wait_pending<0>();
}

// Coarsest level, src/mg/solver.h:264-271: remove the mean of b, then CG
// warm-started from b with the absolute 2-norm stop. One block; only for
// coarsest levels too large for the direct solve of kernels_tail.cu.
template <typename T, int TB = kRedBlock>
__device__ void coarse_cg_block(const Dims& d, T* xv, T* b, T* r, T* p, T* q, double tol, int maxit, int* status) {
    const long long N = d.ncell(), sxy = d.sxy();
    const T off = T(d.n) * T(d.n);
    __shared__ double s_val;
    auto bsum = [&](double v) {
        double a[1] = {v};
        block_sum<1, TB>(a);
        if (threadIdx.x == 0) s_val = a[0];
        __syncthreads();
        return s_val;
    };
    auto apply = [&](const T* in, long long i) {
        const int xi = (int)(i % d.nx), yi = (int)((i % sxy) / d.nx), zi = (int)(i / sxy);
        T S;
        int c;
        // the one-cell (or one-row) levels fold self-neighbours into the diagonal
        lap_row(d, in, xi, yi, zi, S, c);
        return off * (S - lap_count<T>(c) * in[i]);
    };
    double m = 0.0;
    for (long long i = threadIdx.x; i < N; i += blockDim.x) m += (double)b[i];
    m = bsum(m) / (double)N;
    for (long long i = threadIdx.x; i < N; i += blockDim.x) {
        b[i] = b[i] - T(m);
        xv[i] = b[i];
    }
    __syncthreads();
    double rr = 0.0;
    for (long long i = threadIdx.x; i < N; i += blockDim.x) {
        r[i] = b[i] - apply(xv, i);
        p[i] = r[i];
        rr += (double)r[i] * (double)r[i];
    }
    double n0 = bsum(rr);
    int it = 0;
    while (sqrt(n0) > tol) {
        if (it >= maxit || !(n0 == n0)) {
            if (threadIdx.x == 0) status[0] = 3;
            return;
        }
        double pq = 0.0;
        for (long long i = threadIdx.x; i < N; i += blockDim.x) {
            q[i] = apply(p, i);
            pq += (double)p[i] * (double)q[i];
        }
        pq = bsum(pq);
        const T alpha = T(n0 / pq);
        double n1 = 0.0;
        for (long long i = threadIdx.x; i < N; i += blockDim.x) {
            xv[i] = xv[i] + alpha * p[i];
            r[i] = r[i] - q[i] * alpha;
            n1 += (double)r[i] * (double)r[i];
        }
        n1 = bsum(n1);
        const T beta = T(n1 / n0);
        n0 = n1;
        for (long long i = threadIdx.x; i < N; i += blockDim.x) p[i] = p[i] * beta + r[i];
        __syncthreads();
        ++it;
    }
}

template <typename T>
__global__ void __launch_bounds__(kRedBlock) k_coarse_cg(Dims d, T* __restrict__ xv, T* __restrict__ b, T* __restrict__ r,
                                                        T* __restrict__ p, T* __restrict__ q, double tol, int maxit,
                                                        int* status) {
    wait_launch();
    coarse_cg_block(d, xv, b, r, p, q, tol, maxit, status);
}

}  // namespace

__global__ void k_mg_check(cudaGraphConditionalHandle h, MgCheck c, int first) {
    wait_launch();
    const double rms = sqrt(*c.sum) / sqrt(c.n);
    const int done = first ? 0 : *c.cycles + 1;  // after the cycle before this check
    *c.cycles = done;
    cudaGraphSetConditional(h, isfinite(rms) && rms > c.tol && done < c.max ? 1u : 0u);
}
cudaError_t add_mg_check(cudaGraph_t g, cudaGraphConditionalHandle h, MgCheck c, cudaGraphNode_t* node) {
    int first = 1;
    void* args[] = {&h, &c, &first};
    cudaKernelNodeParams p = {};
    p.func = (void*)k_mg_check;
    p.gridDim = dim3(1);
    p.blockDim = dim3(1);
    p.kernelParams = args;
    return cudaGraphAddKernelNode(node, g, nullptr, 0, &p);
}
void launch_mg_check(cudaGraphConditionalHandle h, MgCheck c, cudaStream_t s) { launch_dep(1, 1, 0, s, k_mg_check, h,
        c, 0); }

// smallest level (x extent) on which the smoother and residual take the
// batched z-column kernels, 4 (FP32) or 2 (FP64) cells per thread
// (AFMIB_BATCH_MIN_NX; one cell per thread below). With levels from 96 and from 64 on
// batched, an FP64 channel step at 96x64x64 takes 3.94 and 3.95 ms against 3.83 (its
// colours 10.4 us against 9.9: too few blocks), a mixed step at 96x80x112 3.21 and 3.22
// against 3.26 (7.7 us against 8.4), one at 256^3 14.7 in every case.
int batch_min_nx() {
    static const int v = [] {
        const char* e = std::getenv("AFMIB_BATCH_MIN_NX");
        return e ? std::atoi(e) : 128;
    }();
    return v;
}

template <typename T>
void launch_lap_apply(const Dims& d, T* y, const T* x, cudaStream_t s) {
    AFMIB_IX(d, (launch_dep(grid3(d), dim3(BX, BY), 0, s, k_lap<T, IX>, d, lap_k<T>(d), y, x)));
}
template <typename T>
void launch_residual(const Dims& d, T* r, const T* x, const T* b, RedScratch* sc, double* out, cudaStream_t s, int rev) {
    const LapK<T> k = lap_k<T>(d);
    if (sc && out) {
        const dim3 g = red_grid3(d.nx, d.ny, d.nz, red_target<T>());
        AFMIB_IX(d, (launch_dep(g, dim3(kRBX, kRBY), 0, s, k_residual_norm<T, IX>, d, k, r, x, b, *sc, out)));
    } else if (d.nz % kZU == 0 && d.nx >= batch_min_nx()) {
        const dim3 g((d.nx + BX - 1) / BX, (d.ny + BY - 1) / BY, d.nz / kZU);
        AFMIB_IX(d, (launch_dep(g, dim3(BX, BY), 0, s, k_residual_z2<T, kZU, IX>, d, k, r, x, b, rev)));
    } else {
        AFMIB_IX(d, (launch_dep(grid3(d), dim3(BX, BY), 0, s, k_residual<T, IX>, d, k, r, x, b)));
    }
}
template <typename T>
void launch_residual_red(const Dims& d, T* r, const T* x, const T* b, cudaStream_t s, int rev) {
    constexpr int ZU = 4;
    const int gx = (d.nx / 2 + BX - 1) / BX, gy = (d.ny + BY - 1) / BY;
    const LapK<T> k = lap_k<T>(d);
    if (d.nz % ZU == 0 && d.nx >= batch_min_nx())
        AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz / ZU), dim3(BX, BY), 0, s, k_residual_red<T, ZU, IX>, d, k, r, x,
                                b, rev)));
    else
        AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz), dim3(BX, BY), 0, s, k_residual_red<T, 1, IX>, d, k, r, x, b, rev)));
}
// The pair kernel is opt-in (AFMIB_RBGS_PAIR=1, read at every launch): at
// 256^3 its colour launches took 39.5 us against 29.9 for the scalar kernel
// (53.7 against 56.5 IB steps/s): 60 registers hold it to 4 resident blocks
// and every y-neighbour and b pair brings the other colour's value along.
// Needs full warps along x (nx >= 64) and block rows along y (ny a multiple
// of 8).
constexpr int kPairZU = 4, kPairMinB = 4;
bool rbgs_pair_ok(const Dims& d) {
    const char* e = std::getenv("AFMIB_RBGS_PAIR");
    if (!(e && e[0] == '1')) return false;
    return d.nz > 1 && d.nx >= 2 * BX && d.ny % BY == 0 && d.nz % kPairZU == 0 && ix2_ok(d);
}

// A sweep from x = 0 (x's contents ignored and overwritten). AFMIB_INIT_SWEEP=0: a
// memset of x and the two colours (read at every launch, so that a test can compare
// both in one process).
template <typename T>
void launch_rbgs_first(const Dims& d, T* x, const T* b, cudaStream_t s, double omega, int rev, bool split) {
    if constexpr (sizeof(T) == sizeof(float))
        if (split) {
            launch_dep(dim3(d.nx / 2 / BX, d.ny / BY, d.nz / 4), dim3(BX, BY), 0, s, k_rbgs_first<T, 4, 6, Ix2, true>, d,
                       lap_k<T>(d), T(omega), x, b, rev, T(0));
            return;
        }
    const char* e = std::getenv("AFMIB_INIT_SWEEP");
    if ((e && e[0] == '0') || d.nx % 2) {
        cudaMemsetAsync(x, 0, (size_t)d.ncell() * sizeof(T), s);
        launch_rbgs<T>(d, 0, x, b, s, omega, rev, false);
        launch_rbgs<T>(d, 1, x, b, s, omega, rev, false);
        return;
    }
    if (d.nx < kOmegaMinNx) omega = 1.0;
    constexpr int ZU = 4, MINB = sizeof(T) == sizeof(float) ? 6 : 4;
    const int gx = (d.nx / 2 + BX - 1) / BX, gy = (d.ny + BY - 1) / BY;
    const LapK<T> k = lap_k<T>(d);
    if (d.nz % ZU == 0 && d.nx >= batch_min_nx())
        AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz / ZU), dim3(BX, BY), 0, s, k_rbgs_first<T, ZU, MINB, IX>, d, k,
                                T(omega), x, b, rev, T(0))));
    else
        AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz), dim3(BX, BY), 0, s, k_rbgs_first<T, 1, MINB, IX>, d, k, T(omega),
                                x, b, rev, T(0))));
}

template <typename T>
void launch_rbgs(const Dims& d, int color, T* x, const T* b, cudaStream_t s, double omega, int rev, bool split) {
    if constexpr (sizeof(T) == sizeof(float))
        if (split) {
            launch_dep(dim3(d.nx / 2 / BX, d.ny / BY, d.nz / 4), dim3(BX, BY), 0, s, k_rbgs_split<4, 6>, d, lap_k<T>(d), color,
                       float(omega), x, b, rev);
            return;
        }
    if (d.nx < kOmegaMinNx) omega = 1.0;
    const LapK<T> k = lap_k<T>(d);
    const int gx = (d.nx / 2 + BX - 1) / BX, gy = (d.ny + BY - 1) / BY;
    const dim3 blk(BX, BY);
    constexpr bool f32 = sizeof(T) == sizeof(float);
    if (d.nx >= batch_min_nx() && d.nz % (f32 ? kZU32 : kZU64) == 0) {
        // FP32 on float pairs (opt-in, AFMIB_RBGS_PAIR=1)
        if (f32 && rbgs_pair_ok(d)) {
            const dim3 gp(d.nx / 2 / BX, d.ny / BY, d.nz / kPairZU);
            launch_dep(gp, blk, 0, s, k_rbgs_pair<kPairZU, kPairMinB>, d, color, float(omega), (float*)x,
                       (const float*)b, rev);
            return;
        }
        // FP32: kZU32 z cells per thread, registers capped for 6 resident
        // blocks (50.5 against 50.0 IB steps/s at 256^3 for eight cells
        // and 6 blocks against none; four cells: 29.5 against 30.0 us per
        // 256^3 colour, 61.1 against 60.8 steps/s; 16: spills, two:
        // 32.7 us; four cells with 8 blocks: the same as 6)
        if (f32)
            AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz / kZU32), blk, 0, s, k_rbgs_z2b<T, kZU32, 6, IX>, d, k, color,
                                    T(omega), x, b, rev)));
        else
            AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz / kZU64), blk, 0, s, k_rbgs_z2<T, kZU64, IX>, d, k, color,
                                    T(omega), x, b, rev)));
        return;
    }
    AFMIB_IX(d, (launch_dep(dim3(gx, gy, d.nz), blk, 0, s, k_rbgs<T, IX>, d, k, color, T(omega), x, b)));
}
namespace {
int log2_exact(int v) {
    int k = 0;
    while ((1 << k) < v) ++k;
    return (1 << k) == v ? k : -1;
}
template <typename T>
void* pipe_kernel(int D, bool ch) {
    if (D == 4) return ch ? (void*)k_rbgs_pipe<T, 4, true> : (void*)k_rbgs_pipe<T, 4, false>;
    return ch ? (void*)k_rbgs_pipe<T, 2, true> : (void*)k_rbgs_pipe<T, 2, false>;
}
}  // namespace

template <typename T>
PipeCfg rbgs_pipe_cfg(const Dims& d) {
    PipeCfg c;
    const size_t row = (size_t)d.nx * sizeof(T);
    if (d.nz < 2 || d.nx < 32 || row % 16 != 0) return c;
    if (log2_exact(d.nx) < 0 || log2_exact(d.ny) < 0 || log2_exact(d.nz) < 0) return c;
    constexpr size_t kMaxSmem = 200 * 1024;
    static bool attr = false;
    if (!attr) {
        for (int dd : {4, 2})
            for (bool ch : {false, true})
                if (cudaFuncSetAttribute(pipe_kernel<T>(dd, ch), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kMaxSmem) != cudaSuccess)
                    return c;
        attr = true;
    }
    for (int fy : {4, 2, 1}) {
        if (d.ny % fy) continue;
        for (int dd : {4, 2}) {
            const size_t smem = (size_t)(dd + 4) * (2 * fy + 6) * row;
            if (smem <= kMaxSmem) {
                c.FY = fy;
                c.D = dd;
                c.smem = smem;
                break;
            }
        }
        if (c.FY) break;
    }
    if (!c.FY) return c;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pipe_kernel<T>(c.D, d.channel != 0), kPipeThreads, c.smem);
    if (sms <= 0 || per_sm <= 0) {
        c.FY = 0;
        return c;
    }
    const int resident = sms * per_sm;
    // z chunk: the longest (least redundant halo) that still gives each
    // resident block three or more items
    const int strips = d.ny / c.FY;
    c.ZC = 0;
    for (int zc : {32, 16, 8}) {  // largest first; the smallest dividing one if none reaches 3 items
        if (d.nz % zc) continue;
        c.ZC = zc;
        if ((long long)strips * (d.nz / zc) >= 3LL * resident) break;
    }
    if (!c.ZC) c.ZC = d.nz;  // short z extents: one chunk
    const int items = strips * (d.nz / c.ZC);
    c.grid = items < resident ? items : resident;
    return c;
}

template <typename T>
void launch_rbgs_pipe(const Dims& d, const PipeCfg& c, const T* xin, T* xout, const T* b, int* err, cudaStream_t s) {
    (void)err;  // the copies are cp.async groups: no wait can time out
    const int lnx = log2_exact(d.nx), lny = log2_exact(d.ny);
    if (c.D == 4) {
        if (d.channel) launch_dep(c.grid, kPipeThreads, c.smem, s, k_rbgs_pipe<T, 4, true>, d, xin, xout, b, c.FY,
                                  c.ZC, lnx, lny);
        else launch_dep(c.grid, kPipeThreads, c.smem, s, k_rbgs_pipe<T, 4, false>, d, xin, xout, b, c.FY, c.ZC, lnx,
                        lny);
    } else {
        if (d.channel) launch_dep(c.grid, kPipeThreads, c.smem, s, k_rbgs_pipe<T, 2, true>, d, xin, xout, b, c.FY,
                                  c.ZC, lnx, lny);
        else launch_dep(c.grid, kPipeThreads, c.smem, s, k_rbgs_pipe<T, 2, false>, d, xin, xout, b, c.FY, c.ZC, lnx,
                        lny);
    }
}

// Column-marching transfers (k_restrict_cols, k_prolong_cols) apply to FP32
// 3D power-of-two levels with 32 | nx / 2 (64 for the restriction) and
// kTrBY | ny / 2 and 16-byte aligned fine and coarse arrays;
// AFMIB_TRANSFER_COLS=0 keeps the one-cell kernels (read at every launch, so
// that a test can compare both in one process). FP64 keeps the one-cell
// kernels, which take half of the cells (restrict_after_sweep,
// prolong_before_sweep): residual, restriction and prolongation 119, 136 and 111 us
// per 256^3 launch (21.2, 23.2 and 19.3 at 128^3), against 232, 173 and 193 (35.5,
// 42.1 and 28.7) with the column kernels, which need every cell of the residual, and
// 232, 262 and 147 with one-cell kernels on all cells.
static bool transfer_cols_ok(const Dims& d, const void* fine, const void* coarse) {
    if (const char* e = std::getenv("AFMIB_TRANSFER_COLS"))
        if (e[0] == '0') return false;
    return d.nz > 1 && ix2_ok(d) && (d.nx / 2) % 32 == 0 && (d.ny / 2) % kTrBY == 0 &&
           ((reinterpret_cast<uintptr_t>(fine) | reinterpret_cast<uintptr_t>(coarse)) & 15) == 0;
}
// coarse planes per thread: the largest of 8, 4, 2 that divides the coarse z
// extent and leaves at least AFMIB_TRANSFER_MIN_BLOCKS (default 1024) blocks, else 1
static int transfer_planes(const Dims& d, int bx = 32) {
    const char* e = std::getenv("AFMIB_TRANSFER_MIN_BLOCKS");
    const long long min_blocks = e ? std::atoll(e) : 1024;
    const long long cols = (long long)(d.nx / 2 / bx) * (d.ny / 2 / kTrBY);
    const int cz = d.nz / 2;
    for (int z : {8, 4, 2})
        if (cz % z == 0 && cols * (cz / z) >= min_blocks) return z;
    return 1;
}
inline dim3 transfer_grid(const Dims& d, int planes, int bx = 32) {
    return dim3(d.nx / 2 / bx, d.ny / 2 / kTrBY, d.nz / 2 / planes);
}

template <typename T>
void launch_restrict(const Dims& d, T* coarse, const T* fine, cudaStream_t s, int rev, bool red) {
    if constexpr (sizeof(T) == sizeof(float)) {
        if (!red && transfer_cols_ok(d, fine, coarse) && (d.nx / 2) % TrTile<T>::CX == 0) {
            const int z = transfer_planes(d, TrTile<T>::CX);
            const dim3 g = transfer_grid(d, z, TrTile<T>::CX), b(32, kTrBY);
            if (z == 8) launch_dep(g, b, 0, s, k_restrict_cols<T, 8>, d, coarse, fine, rev);
            else if (z == 4) launch_dep(g, b, 0, s, k_restrict_cols<T, 4>, d, coarse, fine, rev);
            else if (z == 2) launch_dep(g, b, 0, s, k_restrict_cols<T, 2>, d, coarse, fine, rev);
            else launch_dep(g, b, 0, s, k_restrict_cols<T, 1>, d, coarse, fine, rev);
            return;
        }
    }
    dim3 g((d.nx / 2 + BX - 1) / BX, (d.ny / 2 + BY - 1) / BY, d.nz == 1 ? 1 : d.nz / 2);
    if (d.nz > 1)
        AFMIB_IX(d, (red ? launch_dep(g, dim3(BX, BY), 0, s, k_restrict2<T, true, IX>, d, coarse, fine, rev)
                         : launch_dep(g, dim3(BX, BY), 0, s, k_restrict2<T, false, IX>, d, coarse, fine, rev)));
    else
        red ? launch_dep(g, dim3(BX, BY), 0, s, k_restrict<T, true>, d, coarse, fine)
            : launch_dep(g, dim3(BX, BY), 0, s, k_restrict<T, false>, d, coarse, fine);
}
// Fine-level residual and restriction in one pass. AFMIB_RESID_RESTRICT
// (read at every call, so that a test can compare the paths in one process):
// unset or "2": the column kernel (k_resid_restrict_cols) on FP32 levels it
// fits (3D power-of-two, 64 | nx / 2, kTrBY | ny / 2, 16-byte aligned arrays,
// nx >= AFMIB_RR_COLS_MIN_NX, default 256); "1": the ring kernel
// (k_resid_restrict2) on levels with nx >= AFMIB_RESID_RESTRICT_MIN_NX
// (default 256; on smaller levels its grid of 2 RR_T x 2 RR_T fine columns
// per block leaves SMs idle); "0": the residual and restriction kernels.
static int rr_mode(const Dims& d, size_t elem, const void* x, const void* b, const void* cb) {
    const char* e = std::getenv("AFMIB_RESID_RESTRICT");
    const char m = e ? e[0] : '2';
    if (m == '1') {
        const char* mn = std::getenv("AFMIB_RESID_RESTRICT_MIN_NX");
        const int min_nx = mn ? std::atoi(mn) : 256;
        return d.nz > 1 && d.nx >= min_nx && d.nx >= 2 * RR_T && d.ny >= 2 * RR_T && d.nz >= 4 && ix2_ok(d) ? 1 : 0;
    }
    if (m != '2' || elem != sizeof(float)) return 0;
    const char* mn = std::getenv("AFMIB_RR_COLS_MIN_NX");
    const int min_nx = mn ? std::atoi(mn) : 256;
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(b) |
                           reinterpret_cast<uintptr_t>(cb)) & 15) == 0;
    return d.nz > 1 && d.nx >= min_nx && ix2_ok(d) && (d.nx / 2) % 64 == 0 && (d.ny / 2) % kTrBY == 0 && aligned
               ? 2
               : 0;
}
bool resid_restrict_fused_ok(const Dims& d, size_t elem, const void* x, const void* b, const void* cb) {
    return rr_mode(d, elem, x, b, cb) != 0;
}

// An FP32 fine level whose iterate and right-hand side are split by colour: every
// kernel that takes them there has a split form, and the two arrays do not fit in
// the L2 (126 MB): at 512^3 a colour takes 194 us instead of 243, the fused
// residual-restriction 469 instead of 404 and the residual update 1145 instead of 997,
// an IB step 104.6 ms instead of 108.5; at 256^3 26.7 / 29.6, 76 / 65 and 144 / 134 us,
// a step 14.68 / 14.74 ms. AFMIB_SPLIT=0, 1: at no, at every such size.
bool mg_split_ok(const Dims& d, const float* x, const float* b, const float* cb, const float* cx) {
    const char* e = std::getenv("AFMIB_SPLIT");
    if (e ? e[0] == '0' : d.ncell() <= 1ll << 24) return false;
    const char* i = std::getenv("AFMIB_INIT_SWEEP");
    const char* g = std::getenv("AFMIB_UPDATE_DF_GENERIC");
    return !(i && i[0] == '0') && !(g && g[0] == '1') && !rbgs_pair_ok(d) && rr_mode(d, sizeof(float), x, b, cb) == 2 &&
           transfer_cols_ok(d, x, cx) && d.nz % 4 == 0 && d.ny % BY == 0;
}

void mg_kernel_attributes() {
    auto set = [](const void* f) { cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRrSmem); };
    set((const void*)k_resid_restrict_cols<8, false, false>);
    set((const void*)k_resid_restrict_cols<8, false, true>);
    set((const void*)k_resid_restrict_cols<4, false, false>);
    set((const void*)k_resid_restrict_cols<4, false, true>);
    set((const void*)k_resid_restrict_cols<2, false, false>);
    set((const void*)k_resid_restrict_cols<2, false, true>);
    set((const void*)k_resid_restrict_cols<1, false, false>);
    set((const void*)k_resid_restrict_cols<1, false, true>);
    set((const void*)k_resid_restrict_cols<8, true, false>);
    set((const void*)k_resid_restrict_cols<8, true, true>);
    set((const void*)k_resid_restrict_cols<4, true, false>);
    set((const void*)k_resid_restrict_cols<4, true, true>);
    set((const void*)k_resid_restrict_cols<2, true, false>);
    set((const void*)k_resid_restrict_cols<2, true, true>);
    set((const void*)k_resid_restrict_cols<1, true, false>);
    set((const void*)k_resid_restrict_cols<1, true, true>);
}

template <typename T>
void launch_resid_restrict(const Dims& d, T* coarse_b, const T* x, const T* b, cudaStream_t s, int rev,
                           bool red, bool split) {
    if constexpr (sizeof(T) == sizeof(float)) {
        if (split || rr_mode(d, sizeof(T), x, b, coarse_b) == 2) {
            // coarse planes per block: the largest of 8, 4, 2 that leaves at least
            // AFMIB_RR_MIN_BLOCKS (default 512) blocks (two resident per SM)
            const char* e = std::getenv("AFMIB_RR_MIN_BLOCKS");
            const long long min_blocks = e ? std::atoll(e) : 512;
            const long long cols = (long long)(d.nx / 2 / 64) * (d.ny / 2 / kTrBY);
            const int cz = d.nz / 2;
            int z = 1;
            for (int c : {8, 4, 2})
                if (cz % c == 0 && cols * (cz / c) >= min_blocks) {
                    z = c;
                    break;
                }
            const dim3 g(d.nx / 2 / 64, d.ny / 2 / kTrBY, cz / z), blk(32, kTrBY);
            float* cbf = reinterpret_cast<float*>(coarse_b);
            const float* xf = reinterpret_cast<const float*>(x);
            const float* bf = reinterpret_cast<const float*>(b);
#define AFMIB_RR_COLS(CZV)                                                                            \
    do {                                                                                              \
        if (d.channel && split)                                                                       \
            launch_dep(g, blk, kRrSmem, s, k_resid_restrict_cols<CZV, true, true>, d, cbf, xf, bf, rev); \
        else if (split)                                                                               \
            launch_dep(g, blk, kRrSmem, s, k_resid_restrict_cols<CZV, false, true>, d, cbf, xf, bf, rev); \
        else if (d.channel)                                                                           \
            launch_dep(g, blk, kRrSmem, s, k_resid_restrict_cols<CZV, true, false>, d, cbf, xf, bf, rev); \
        else                                                                                          \
            launch_dep(g, blk, kRrSmem, s, k_resid_restrict_cols<CZV, false, false>, d, cbf, xf, bf, rev); \
    } while (0)
            if (z == 8) AFMIB_RR_COLS(8);
            else if (z == 4) AFMIB_RR_COLS(4);
            else if (z == 2) AFMIB_RR_COLS(2);
            else AFMIB_RR_COLS(1);
#undef AFMIB_RR_COLS
            return;
        }
    }
    // the ring kernel: coarse planes per block 8 where that still gives two
    // blocks per SM, else 2
    const int cols = (d.nx / 2 / RR_T) * (d.ny / 2 / RR_T), cz = d.nz / 2;
    if (cz % 8 == 0 && cols * (cz / 8) >= 2 * 152)
        launch_dep(dim3(d.nx / 2 / RR_T, d.ny / 2 / RR_T, cz / 8), RR_THREADS, 0, s, k_resid_restrict2<T, 8>, d,
                   coarse_b, x, b, rev, red);
    else
        launch_dep(dim3(d.nx / 2 / RR_T, d.ny / 2 / RR_T, cz / 2), RR_THREADS, 0, s, k_resid_restrict2<T, 2>, d,
                   coarse_b, x, b, rev, red);
}

template <typename T>
void launch_prolong_add(const Dims& d, T* fine, const T* coarse, cudaStream_t s, int rev, bool black, bool split) {
    if constexpr (sizeof(T) == sizeof(float)) {
        if (split || transfer_cols_ok(d, fine, coarse)) {
            // AFMIB_PROLONG_MAX_PLANES caps the planes per block (a sweep knob)
            const char* e = std::getenv("AFMIB_PROLONG_MAX_PLANES");
            int z = std::min(transfer_planes(d), e ? std::max(1, std::atoi(e)) : 8);
            while (z & (z - 1)) z &= z - 1;  // a power of two, so a divisor of the plane count
            const dim3 g = transfer_grid(d, z), b(32, kTrBY);
            if (z == 8) launch_dep(g, b, 0, s, split ? k_prolong_cols<T, 8, true> : k_prolong_cols<T, 8, false>, d, fine, coarse, rev);
            else if (z == 4) launch_dep(g, b, 0, s, split ? k_prolong_cols<T, 4, true> : k_prolong_cols<T, 4, false>, d, fine, coarse, rev);
            else if (z == 2) launch_dep(g, b, 0, s, split ? k_prolong_cols<T, 2, true> : k_prolong_cols<T, 2, false>, d, fine, coarse, rev);
            else launch_dep(g, b, 0, s, split ? k_prolong_cols<T, 1, true> : k_prolong_cols<T, 1, false>, d, fine, coarse, rev);
            return;
        }
    }
    dim3 g((d.nx / 2 + BX - 1) / BX, (d.ny / 2 + BY - 1) / BY, d.nz == 1 ? 1 : d.nz / 2);
    if (d.nz > 1)
        AFMIB_IX(d, (black ? launch_dep(g, dim3(BX, BY), 0, s, k_prolong2<T, true, true, IX>, d, fine, coarse, rev)
                           : launch_dep(g, dim3(BX, BY), 0, s, k_prolong2<T, true, false, IX>, d, fine, coarse, rev)));
    else
        black ? launch_dep(g, dim3(BX, BY), 0, s, k_prolong<T, true, true>, d, fine, coarse)
              : launch_dep(g, dim3(BX, BY), 0, s, k_prolong<T, true, false>, d, fine, coarse);
}
template <typename T>
void launch_prolong_assign(const Dims& d, T* fine, const T* coarse, cudaStream_t s) {
    dim3 g((d.nx / 2 + BX - 1) / BX, (d.ny / 2 + BY - 1) / BY, d.nz == 1 ? 1 : d.nz / 2);
    if (d.nz > 1) AFMIB_IX(d, (launch_dep(g, dim3(BX, BY), 0, s, k_prolong2<T, false, false, IX>, d, fine, coarse, 0)));
    else launch_dep(g, dim3(BX, BY), 0, s, k_prolong<T, false, false>, d, fine, coarse);
}
template <typename TD>
void launch_lap_defect(const Dims& d, TD* r, const double* x, const double* b, RedScratch sc, double* out, cudaStream_t s,
                       float* r_lo) {
    launch_dep(red_grid3(d.nx, d.ny, d.nz), dim3(kRBX, kRBY), 0, s, k_lap_defect<TD>, d, lap_k<double>(d), r, x, b,
               sc, out, r_lo, lo_split());
}
void launch_lap_defect_df(const Dims& d, float* rh, float* rl, const double* x, const double* b, const double* sum,
                          double scale, RedScratch sc, double* out, cudaStream_t s, bool split) {
    const dim3 blk(kRBX, kRBY);
    if (split) {
        launch_dep(red_grid3(d.nx, d.ny, d.nz / 2), blk, 0, s, k_lap_defect_df<2, Ix2, true>, d, rh, rl, x, b, sum, scale, sc,
                   out);
        return;
    }
    if (d.nz % 2 == 0)
        AFMIB_IX(d, (launch_dep(red_grid3(d.nx, d.ny, d.nz / 2), blk, 0, s, k_lap_defect_df<2, IX, false>, d, rh, rl, x, b,
                                sum, scale, sc, out)));
    else
        AFMIB_IX(d, (launch_dep(red_grid3(d.nx, d.ny, d.nz), blk, 0, s, k_lap_defect_df<1, IX, false>, d, rh, rl, x, b, sum,
                                scale, sc, out)));
}
void launch_lap_update_df(const Dims& d, double* x, const float* e, float* rh, float* rl, RedScratch sc, double* out,
                          cudaStream_t s, bool split) {
    constexpr int ZU = 2;
    const char* g = std::getenv("AFMIB_UPDATE_DF_GENERIC");
    if (split || (d.nz > 1 && d.nz % ZU == 0 && !(g && g[0] == '1'))) {
        const int gx = (d.nx + kRBX - 1) / kRBX, gy = (d.ny + kRBY - 1) / kRBY;
        int gz = d.nz / ZU;
        if ((long long)gx * gy * gz > kMaxRedBlocks) gz = std::max(1, kMaxRedBlocks / (gx * gy));
        if (split) {
            launch_dep(dim3(gx, gy, gz), dim3(kRBX, kRBY), 0, s, k_lap_update_df2<ZU, kUpdateMinBlocks, Ix2, true>, d, x, e,
                       rh, rl, sc, out);
            return;
        }
        AFMIB_IX(d, (launch_dep(dim3(gx, gy, gz), dim3(kRBX, kRBY), 0, s, k_lap_update_df2<ZU, kUpdateMinBlocks, IX, false>,
                                d, x, e, rh, rl, sc, out)));
        return;
    }
    launch_dep(red_grid3(d.nx, d.ny, d.nz), dim3(kRBX, kRBY), 0, s, k_lap_update_df, d, x, e, rh, rl, sc, out);
}
bool launch_lap_defect_bfp(const Dims& d, float* r, const double* x, const double* b, RedScratch sc, double* out,
                           cudaStream_t s) {
    int k = 0;
    while ((1 << k) < d.n) ++k;
    if ((1 << k) != d.n || 2 * k > 126) return false;  // n must be a power of two
    launch_dep(red_grid3(d.nx, d.ny, d.nz), dim3(kRBX, kRBY), 0, s, k_lap_defect_bfp, d, 2 * k, r, x, b, sc, out);
    return true;
}
template void launch_lap_defect<float>(const Dims&, float*, const double*, const double*, RedScratch, double*,
                                       cudaStream_t, float*);

template <typename T>
void launch_coarse_solve(const Dims& d, T* x, T* b, T* r, T* p, T* q, double tol, int maxit, int* status, cudaStream_t s) {
    launch_dep(1, kRedBlock, 0, s, k_coarse_cg<T>, d, x, b, r, p, q, tol, maxit, status);
}

#define AFMIB_MG_INST(T)                                                                                 \
    template void launch_lap_apply<T>(const Dims&, T*, const T*, cudaStream_t);                          \
    template void launch_residual<T>(const Dims&, T*, const T*, const T*, RedScratch*, double*, cudaStream_t, int); \
    template void launch_residual_red<T>(const Dims&, T*, const T*, const T*, cudaStream_t, int);                  \
    template void launch_rbgs<T>(const Dims&, int, T*, const T*, cudaStream_t, double, int, bool);                        \
    template void launch_rbgs_first<T>(const Dims&, T*, const T*, cudaStream_t, double, int, bool);                      \
    template PipeCfg rbgs_pipe_cfg<T>(const Dims&);                                                      \
    template void launch_rbgs_pipe<T>(const Dims&, const PipeCfg&, const T*, T*, const T*, int*, cudaStream_t); \
    template void launch_restrict<T>(const Dims&, T*, const T*, cudaStream_t, int, bool);                   \
    template void launch_prolong_add<T>(const Dims&, T*, const T*, cudaStream_t, int, bool, bool);                \
    template void launch_resid_restrict<T>(const Dims&, T*, const T*, const T*, cudaStream_t, int, bool, bool); \
    template void launch_prolong_assign<T>(const Dims&, T*, const T*, cudaStream_t);                     \
    template void launch_coarse_solve<T>(const Dims&, T*, T*, T*, T*, T*, double, int, int*, cudaStream_t);

AFMIB_MG_INST(double)
AFMIB_MG_INST(float)

}  // namespace afmib
