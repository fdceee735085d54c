// Multigrid tail: the V-cycle below a level of at most kTailCells cells (32^3,
// or a 2D grid of 128 x 256 cells) in one launch on one thread-block cluster.
//
// The coarse levels are a few thousand cells, so a launch per phase costs more
// than the phase, and one block is bound by the shared-memory latency of its
// 45 phases in FP32 and by one SM's FP64 pipe in FP64. Here a cluster of up to
// 16 CTAs holds every level in distributed shared memory: a CTA owns a slab of
// z planes (rows of y on a 2D grid) of each level, reads the neighbouring
// slabs' planes through the cluster's shared-memory window, and cluster
// barriers separate the phases; the levels too small to share (at most
// kLocalCells cells) stay in the first CTA with block barriers. The coarsest
// level is solved directly in FP64 in the tensor-product eigenbasis of its
// Laplacian (six short dense transforms), with the constant mode dropped: what
// the mean removal and CG of src/mg/solver.h:264-271 converge to.
//
// Every cell takes the level kernels' expressions with the same terms in the
// same order (lap_row, rbgs_cell, restrict_cell, prolong_cell of
// kernels_mg.cu), so the V-cycle equals the launch-by-launch one bit for bit.
//
// Measured on GB300 (us per launch, launches back to back; before: one block of
// 512 threads from 16^3, general indices and a one-block CG on the coarsest
// level elsewhere): FP64 from 16^3 44 (was 121), FP32 from 32^3 39 (was 40 from
// 16^3 plus 16 for the 32^3 level's launches), FP64 2D from 128^2 69 (was 133
// from 64^2 plus 28), a coarsest 15^3 level with the 30^3 above it 35 (was 630).
// The phases are bound by latency: a cluster barrier takes 480 clocks, a load
// from another CTA's shared memory 255 (local: 51), a dependent FP64
// instruction 64 and one SM issues an FP64 warp instruction every 16-19.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "kernels.h"
#include "mg_cells.cuh"

namespace cg = cooperative_groups;

namespace afmib {

namespace {

constexpr int kTailThreads = 512;
constexpr size_t kTailSmem = 200 * 1024;
constexpr int kLaneCells = 64;   // coarse cells per CTA up to which the restriction takes a half warp per cell

// One level of the tail. On a 2D grid the slabs are rows: ny = 1 and nz is the
// grid's y extent (flat).
template <typename T>
struct TailLv {
    int nx, ny, nz;
    int P, nc;                        // planes per CTA (1, even, or all), CTAs that own any
    unsigned mP, mhx, mny, mcy;       // division by P, nx/2, ny and ny/2 (fdiv)
    int ox, ob, orr;                  // offsets of x, b, r in every CTA's shared memory, in T
    int nu1, nu2, red, black;         // restrict_after_sweep, prolong_before_sweep
    T omega, inv, off;                // off = n^2 and inv = 1 / n^2, as the level kernels round them
};
template <typename T>
struct TailArgs {
    TailLv<T> lv[kMaxTailLevels];
    int nlev, flat, channel, x_zero;
    int ofa, ofb;  // the coarsest solve's two FP64 vectors, in doubles
    T* gx;
    const T* gb;
    const double *vx, *vy, *vz, *lx, *ly, *lz;  // eigenvectors (row k: mode k) and eigenvalues per axis
    double n2;                                  // the coarsest level's n^2
    int* status;
};

// floor(e / d) for e * d < 2^32, m = ceil(2^32 / d) (0: d = 1)
__device__ __forceinline__ int fdiv(int e, unsigned m) { return m ? (int)__umulhi((unsigned)e, m) : e; }
inline unsigned fdiv_magic(int d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }

// shared-memory pointer of plane z of an array that starts at `base` in every CTA
template <typename T, typename U>
__device__ __forceinline__ U* plane_of(U* base, const TailLv<T>& L, int z, int rank) {
    const int own = L.nc == 1 ? 0 : fdiv(z, L.mP);
    U* p = own == rank ? base : cg::this_cluster().map_shared_rank(base, own);
    return p + (z - own * L.P) * (L.nx * L.ny);
}

// shared-memory accesses by 32-bit address: of this CTA's window (lds, sts) or
// of any CTA's in the cluster (ldc)
__device__ __forceinline__ float lds(unsigned a, float) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double lds(unsigned a, double) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float ldc(unsigned a, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double ldc(unsigned a, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts(unsigned a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ unsigned mapa(unsigned a, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// One cell of x and its neighbours as shared-memory addresses (ym, yp: 0 beyond
// a channel wall; zm, zp: bit 0 set in another CTA's window, whose loads take
// five times a local one and a path of their own). A thread keeps the cells it updates in registers for all the
// sweeps and the residual of a level: decoding them again in every phase was
// more than half of a phase of a few hundred cells.
struct Cell {
    unsigned c, xm, xp, ym, yp, zm, zp;
};
constexpr int kCells = 2;  // cells per colour and thread; larger slabs take passes of them

// the e-th cell of a colour of the CTA's slab
template <typename T, bool FLAT, bool CH>
__device__ __forceinline__ Cell cell_of(const TailLv<T>& L, unsigned x0, int z0, int pn, int rank, int color, int e) {
    const int nx = L.nx, ny = L.ny, sxy = nx * ny;
    const int row = fdiv(e, L.mhx), t = e - row * (nx >> 1);
    const int zl = FLAT ? row : fdiv(row, L.mny), y = FLAT ? 0 : row - zl * ny;
    const int x = 2 * t + ((y + z0 + zl + color) & 1), i = x + nx * row;
    const unsigned sz = sizeof(T);
    Cell q;
    q.c = x0 + sz * i;
    q.xm = x0 + sz * (x == 0 ? i + nx - 1 : i - 1);
    q.xp = x0 + sz * (x == nx - 1 ? i - (nx - 1) : i + 1);
    q.ym = q.yp = 0;
    if (!FLAT) {
        if (y > 0) q.ym = x0 + sz * (i - nx);
        else if (!CH) q.ym = x0 + sz * (i + sxy - nx);
        if (y < ny - 1) q.yp = x0 + sz * (i + nx);
        else if (!CH) q.yp = x0 + sz * (i - (sxy - nx));
    }
    // plane z of the slab or of the neighbouring CTA's
    auto plane = [&](int z) {
        const int own = L.nc == 1 ? 0 : fdiv(z, L.mP);
        const unsigned a = x0 + sz * (i - zl * sxy + (z - own * L.P) * sxy);
        return L.nc == 1 || own == rank ? a : mapa(a, own) | 1u;
    };
    const int z = z0 + zl;
    q.zm = zl > 0 ? q.c - sz * sxy : plane(z == 0 ? L.nz - 1 : z - 1);
    q.zp = zl < pn - 1 ? q.c + sz * sxy : plane(z == L.nz - 1 ? 0 : z + 1);
    return q;
}

template <typename T, bool DIST>
__device__ __forceinline__ T ldz(unsigned a) {
    if (DIST && (a & 1u)) return ldc(a & ~1u, T(0));
    return lds(a, T(0));
}
// neighbour sum and count: lap_row's terms in its order
template <typename T, bool FLAT, bool CH, bool DIST>
__device__ __forceinline__ T neighbours(const Cell& q, int& c) {
    const T z = T(0);
    T S = (lds(q.xm, z) + lds(q.xp, z)) + (ldz<T, DIST>(q.zm) + ldz<T, DIST>(q.zp));
    c = FLAT ? 4 : 6;
    if (!FLAT) {
        if (CH) {
            if (q.ym) S += lds(q.ym, z); else --c;
            if (q.yp) S += lds(q.yp, z); else --c;
        } else {
            S += lds(q.ym, z) + lds(q.yp, z);
        }
    }
    return S;
}

// Gauss-Seidel value of one cell (rbgs_cell's arithmetic); db: bytes from x to b
template <typename T, bool FLAT, bool CH, bool DIST>
__device__ __forceinline__ T gs_cell(const Cell& q, unsigned db, T inv, T omega) {
    int c;
    const T S = neighbours<T, FLAT, CH, DIST>(q, c);
    const T rc = FLAT || (CH && c == 4) ? T(0.25) : (CH && c == 5 ? T(1.0 / 5.0) : T(1.0 / 6.0));
    T v = (S - lds(q.c + db, T(0)) * inv) * rc;
    if (omega != T(1)) v = v + (omega - T(1)) * (v - lds(q.c, T(0)));
    return v;
}

// The nu sweeps of a level and, with RES, the residual r = b - L x after them:
// two cells per thread and colour in registers where the slab's colours fit,
// else decoded pass by pass. Every load of a thread's cells of a colour comes
// before their stores (a colour reads the other colour and itself only).
// (Functions of their own, not inlined at their call sites: the kernel runs
// each phase a few times on one block per SM, and inlined copies spilled
// registers and missed the instruction cache.)
template <typename T, bool FLAT, bool CH, bool DIST>
__device__ __noinline__ void smooth(const TailLv<T>& L, unsigned x0, int z0, int pn, int rank, int nu, bool res) {
    auto barrier = []() {
        if constexpr (DIST) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int total = pn * L.ny * (L.nx >> 1), bd = blockDim.x, tid = threadIdx.x;
    const unsigned db = (unsigned)sizeof(T) * (unsigned)(L.ob - L.ox), dr = (unsigned)sizeof(T) * (unsigned)(L.orr - L.ox);
    const T inv = L.inv, omega = L.omega, off = L.off;
    auto update = [&](const Cell (&q)[kCells], int n) {
        T v[kCells];
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (k < n) v[k] = gs_cell<T, FLAT, CH, DIST>(q[k], db, inv, omega);
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (k < n) sts(q[k].c, v[k]);
    };
    auto resid = [&](const Cell (&q)[kCells], int n) {
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (k < n) {
                int c;
                const T S = neighbours<T, FLAT, CH, DIST>(q[k], c);
                const T cc = FLAT || (CH && c == 4) ? T(4) : (CH && c == 5 ? T(5) : T(6));
                sts(q[k].c + dr, lds(q[k].c + db, T(0)) - off * (S - cc * lds(q[k].c, T(0))));
            }
    };
    auto decode = [&](Cell (&q)[kCells], int color, int e) {
        int n = 0;
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (e + k * bd < total) {
                q[k] = cell_of<T, FLAT, CH>(L, x0, z0, pn, rank, color, e + k * bd);
                n = k + 1;
            }
        return n;
    };
    if (total <= kCells * bd) {
        Cell red[kCells], black[kCells];
        const int nr = decode(red, 0, tid), nb = decode(black, 1, tid);
        for (int j = 0; j < nu; ++j) {
            update(red, nr);
            barrier();
            update(black, nb);
            barrier();
        }
        if (res) {
            resid(red, nr);
            if (L.red) {
#pragma unroll
                for (int k = 0; k < kCells; ++k)
                    if (k < nb) sts(black[k].c + dr, T(0));
            } else {
                resid(black, nb);
            }
            barrier();
        }
        return;
    }
    Cell q[kCells];
    for (int j = 0; j < 2 * nu; ++j) {
        for (int e = tid; e < total; e += kCells * bd) update(q, decode(q, j & 1, e));
        barrier();
    }
    if (res) {
        for (int color = 0; color < 2; ++color)
            for (int e = tid; e < total; e += kCells * bd) {
                const int n = decode(q, color, e);
                if (color == 0 || !L.red) {
                    resid(q, n);
                } else {
#pragma unroll
                    for (int k = 0; k < kCells; ++k)
                        if (k < n) sts(q[k].c + dr, T(0));
                }
            }
        barrier();
    }
}

// Full weighting of the CTA's share of the coarse cells: the coarse planes
// whose two fine planes it owns, or half the cells of one where it owns a
// single fine plane (the other owner takes the other half). The coarse x starts
// at zero.
template <typename T, bool FLAT, bool CH>
__device__ __noinline__ void restrict_share(const TailLv<T>& L, const TailLv<T>& C, T* R, T* cb, T* cx, int z0,
                                               int pn, int rank) {
    const int nx = L.nx, ny = L.ny, nz = L.nz, hx = nx >> 1, cxy = C.nx * C.ny;
    const bool half = L.P == 1;
    const int first = half && (z0 & 1) ? cxy / 2 : 0;
    const int total = pn == 0 ? 0 : (half ? ((z0 & 1) ? cxy : cxy / 2) : (pn >> 1) * cxy);
    // coarse cell e: its taps' planes, columns and rows, and where it goes
    auto where = [&](int e, int& xc, int& yc, int& zc, int& p) {
        const int row = fdiv(e, L.mhx);
        xc = e - row * hx;
        const int zl = FLAT ? row : (half ? 0 : fdiv(row, L.mcy));
        yc = FLAT ? 0 : row - zl * (ny >> 1);
        zc = (z0 >> 1) + zl;
        p = e - zl * cxy;
    };
    auto plane = [&](int zc, int k) -> const T* {
        const int zz = 2 * zc - 1 + k;
        return plane_of<T>(R, L, zz < 0 ? zz + nz : (zz >= nz ? zz - nz : zz), rank);
    };
    auto col = [&](int xc, int k) {
        const int xx = 2 * xc - 1 + k;
        return xx < 0 ? xx + nx : (xx >= nx ? xx - nx : xx);
    };
    auto rowof = [&](int yc, int k) {
        const int yy = 2 * yc - 1 + k;
        if (CH) return nx * (yy < 0 ? 0 : (yy > ny - 1 ? ny - 1 : yy));
        return nx * (yy < 0 ? yy + ny : (yy >= ny ? yy - ny : yy));
    };
    auto store = [&](int zc, int p, T acc) {
        plane_of<T>(cb, C, zc, rank)[p] = acc;
        plane_of<T>(cx, C, zc, rank)[p] = T(0);
    };
    if (!FLAT && total - first <= kLaneCells) {
        // few cells: a half warp per cell, a row of four taps per lane, the row
        // and plane sums through shuffles (one SM quarter issues an FP64 warp
        // instruction every 64 clocks: 9 of them instead of 63 in a row)
        const int lane = threadIdx.x & 31, kz = (lane >> 2) & 3, ky = lane & 3, base = lane & 16;
        const int hw = threadIdx.x >> 4, nhw = blockDim.x >> 4;
        for (int r = first; r < total; r += nhw) {
            const int e = r + hw;
            T rs = T(0);
            int xc = 0, yc = 0, zc = 0, p = 0;
            if (e < total) {
                where(e, xc, yc, zc, p);
                const T* q = plane(zc, kz) + rowof(yc, ky);
                rs = full4<T>(q[col(xc, 0)], q[col(xc, 1)], q[col(xc, 2)], q[col(xc, 3)]);  // black taps are zeros
            }
            T s[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) s[k] = __shfl_sync(0xffffffffu, rs, base | (kz << 2) | k);
            const T ps = full4<T>(s[0], s[1], s[2], s[3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) s[k] = __shfl_sync(0xffffffffu, ps, base | (k << 2));
            if (e < total && (lane & 15) == 0) store(zc, p, full4<T>(s[0], s[1], s[2], s[3]) * T(1.0 / 512.0));
        }
        return;
    }
    for (int e = first + threadIdx.x; e < total; e += blockDim.x) {
        int xc, yc, zc, p;
        where(e, xc, yc, zc, p);
        const T* rp[4];
        int xs[4], ys[4];
        unsigned odd = 0;  // parity of row ky (clamped at channel walls)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            rp[k] = plane(zc, k);
            xs[k] = col(xc, k);
            ys[k] = rowof(yc, k);
            odd |= (unsigned)((fdiv(ys[k], L.mhx) >> 1) & 1) << k;  // ys = nx y
        }
        T acc;
        if (!FLAT && L.red)
            acc = restrict_rows<T>([&](int kz, int ky) {
                // plane 2 zc - 1 + kz: the parity of kz + 1
                return red_row<T>((((odd >> ky) + kz + 1) & 1) != 0,
                                  [&](int kx) { return rp[kz][xs[kx] + ys[ky]]; });
            });
        else if (FLAT) acc = restrict_plane<T>([&](int ky, int kx) { return rp[ky][xs[kx]]; }) * T(1.0 / 64.0);
        else acc = restrict_taps<T>([&](int kz, int ky, int kx) { return rp[kz][xs[kx] + ys[ky]]; });
        store(zc, p, acc);
    }
}

// x += P xc on the CTA's planes: fine plane z = 2 zc + 1 is the first (nearest
// to zc) and 2 zc + 2 the second (nearest to zc + 1) of a coarse pair
template <typename T, bool FLAT, bool CH>
__device__ __noinline__ void prolong_share(const TailLv<T>& L, const TailLv<T>& C, T* X, const T* cx, int z0, int pn,
                                              int rank) {
    const int nx = L.nx, ny = L.ny, sxy = nx * ny, hx = C.nx, cy = C.ny, total = pn * hx * cy;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int row = fdiv(e, L.mhx), xc = e - row * hx;
        const int zl = FLAT ? row : fdiv(row, L.mcy), yc = FLAT ? 0 : row - zl * cy;
        const int z = z0 + zl, zc = z == 0 ? C.nz - 1 : (z - 1) >> 1, zn = zc + 1 == C.nz ? 0 : zc + 1;
        const T* p = plane_of<T>(cx, C, zc, rank);
        const T* q = plane_of<T>(cx, C, zn, rank);
        const T* near = (z & 1) ? p : q;
        const T* far = (z & 1) ? q : p;
        const int xn = xc + 1 == hx ? 0 : xc + 1;
        const int xf[2] = {2 * xc + 1, 2 * xc + 2 == nx ? 0 : 2 * xc + 2};
        T* Xp = X + zl * sxy;
        auto put = [&](int x, int y, T v, T s) {
            const int i = x + nx * y;
            Xp[i] = fma_t(v, s, Xp[i]);
        };
        const bool black = L.black;
        const int rz = (z & 1) ? 0 : 1;  // on a 2D grid z is y
        if (FLAT) {
            prolong_row2(near[xc], near[xn], far[xc], far[xn], black_col(black, rz, 1), [&](int rx, T v, T s) { put(xf[rx], 0, v, s); });
            continue;
        }
        const int a = hx * yc;
        if (!CH || yc < cy - 1) {
            const int b = yc + 1 == cy ? 0 : a + hx;
            const int yf[2] = {2 * yc + 1, 2 * yc + 2 == ny ? 0 : 2 * yc + 2};
            prolong_plane4(near[xc + a], near[xn + a], near[xc + b], near[xn + b], far[xc + a], far[xn + a],
                           far[xc + b], far[xn + b], black, rz, [&](int rx, int ry, T v, T s) { put(xf[rx], yf[ry], v, s); });
        }
        if (CH && yc == 0)
            prolong_row2(near[xc + a], near[xn + a], far[xc + a], far[xn + a], black_col(black, 1, rz),
                         [&](int rx, T v, T s) { put(xf[rx], 0, v, s); });
        if (CH && yc == cy - 1)
            prolong_row2(near[xc + a], near[xn + a], far[xc + a], far[xn + a], black_col(black, 0, rz),
                         [&](int rx, T v, T s) { put(xf[rx], ny - 1, v, s); });
    }
}

// out[.., k, ..] = sum_j M[k][j] in[.., j, ..] along x (AX 0) or y (AX 1) of
// the CTA's planes; fwd: M = V, else V^T
template <int AX>
__device__ __forceinline__ void transform(const double* in, double* out, const double* __restrict__ V, bool fwd, int nx,
                                          int ny, int total) {
    const int m = AX == 0 ? nx : ny, st = AX == 0 ? 1 : nx;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int k = AX == 0 ? e % nx : (e / nx) % ny;
        const double* p = in + (e - k * st);
        double s = 0.0;
        if (fwd)
            for (int j = 0; j < m; ++j) s += __ldg(V + k * m + j) * p[j * st];
        else
            for (int j = 0; j < m; ++j) s += __ldg(V + j * m + k) * p[j * st];
        out[e] = s;
    }
}

template <typename T, bool FLAT, bool CH>
__global__ void __launch_bounds__(kTailThreads, 1) k_mg_tail(const __grid_constant__ TailArgs<T> args) {
    extern __shared__ __align__(16) unsigned char tsm[];
    T* const sm = (T*)tsm;
    // the level tables in shared memory: read through the constant bank, each
    // level's first phase waited about 2500 clocks for them
    __shared__ TailArgs<T> g;
    for (int i = threadIdx.x; i < (int)(sizeof(g) / sizeof(int)); i += blockDim.x)
        reinterpret_cast<int*>(&g)[i] = reinterpret_cast<const int*>(&args)[i];
    __syncthreads();
    const cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    auto own = [&](const TailLv<T>& L, int& z0) {
        z0 = rank * L.P;
        const int n = L.nz - z0;
        return rank >= L.nc ? 0 : (n < L.P ? n : L.P);
    };
    auto barrier = [&](const TailLv<T>& L) {
        if (L.nc > 1) cl.sync();
        else __syncthreads();
    };
    {
        const TailLv<T>& L = g.lv[0];
        int z0;
        const int pn = own(L, z0), total = pn * L.nx * L.ny;
        const T* gb = g.gb + (size_t)z0 * L.nx * L.ny;
        const T* gx = g.gx + (size_t)z0 * L.nx * L.ny;
        for (int i = threadIdx.x; i < total; i += 4 * blockDim.x) {  // four loads in flight per array
            T vb[4], vx[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = i + k * blockDim.x;
                vb[k] = j < total ? gb[j] : T(0);
                vx[k] = j < total && !g.x_zero ? gx[j] : T(0);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = i + k * blockDim.x;
                if (j < total) {
                    sm[L.ob + j] = vb[k];
                    sm[L.ox + j] = vx[k];
                }
            }
        }
        barrier(L);
    }
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(sm);
    auto smooth_level = [&](const TailLv<T>& L, int nu, bool res) {
        int z0;
        const int pn = own(L, z0);
        const unsigned x0 = sbase + (unsigned)sizeof(T) * (unsigned)L.ox;
        if (L.nc > 1) smooth<T, FLAT, CH, true>(L, x0, z0, pn, rank, nu, res);
        else smooth<T, FLAT, CH, false>(L, x0, z0, pn, rank, nu, res);
    };
    const int last = g.nlev - 1;
    // a coarsest level of one cell corrects nothing (its solution is the
    // dropped constant): the transfers to and from it are left out too
    const bool one = g.lv[last].nx * g.lv[last].ny * g.lv[last].nz == 1;
    for (int l = 0; l < last; ++l) {
        const TailLv<T>& L = g.lv[l];
        if (L.nc == 1 && rank != 0) break;  // the first CTA's own levels
        const TailLv<T>& C = g.lv[l + 1];
        const bool down = !(one && l + 1 == last);
        smooth_level(L, L.nu1, down);
        if (!down) break;
        int z0;
        const int pn = own(L, z0);
        restrict_share<T, FLAT, CH>(L, C, sm + L.orr, sm + C.ob, sm + C.ox, z0, pn, rank);
        barrier(L);
    }
    // coarsest level: V^T diag(1 / lambda) V b over the three axes, the
    // constant mode dropped; rows of fixed-order FP64 sums
    if (one) {
        if (last == 0 && rank == 0 && threadIdx.x == 0) sm[g.lv[0].ox] = T(0);
        if (last == 0) __syncthreads();
    } else if (g.lv[last].nc > 1 || rank == 0) {
        const TailLv<T>& L = g.lv[last];
        int z0;
        const int pn = own(L, z0), nx = L.nx, ny = L.ny, nz = L.nz, sxy = nx * ny, total = pn * sxy;
        double *A = (double*)tsm + g.ofa, *D = (double*)tsm + g.ofb;
        T* X = sm + L.ox;
        const T* B = sm + L.ob;
        for (int i = threadIdx.x; i < total; i += blockDim.x) A[i] = (double)B[i];
        __syncthreads();
        transform<0>(A, D, g.vx, true, nx, ny, total);
        __syncthreads();
        transform<1>(D, A, g.vy, true, nx, ny, total);
        barrier(L);
        const double n2 = g.n2;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            const int zl = e / sxy, p = e - zl * sxy, ky = p / nx, kx = p - ky * nx, kz = z0 + zl;
            double s = 0.0;
            for (int j = 0; j < nz; ++j) s += __ldg(g.vz + kz * nz + j) * plane_of<T>(A, L, j, rank)[p];
            if (kx + ky + kz == 0) {
                if (!isfinite(s)) atomicExch(g.status, 3);
                D[e] = 0.0;
            } else {
                D[e] = s / (n2 * ((g.lx[kx] + g.ly[ky]) + g.lz[kz]));
            }
        }
        barrier(L);
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            const int zl = e / sxy, p = e - zl * sxy, z = z0 + zl;
            double s = 0.0;
            for (int k = 0; k < nz; ++k) s += __ldg(g.vz + k * nz + z) * plane_of<T>(D, L, k, rank)[p];
            A[e] = s;
        }
        barrier(L);  // D is read by its neighbours until here
        transform<1>(A, D, g.vy, false, nx, ny, total);
        __syncthreads();
        transform<0>(D, A, g.vx, false, nx, ny, total);
        __syncthreads();
        for (int i = threadIdx.x; i < total; i += blockDim.x) X[i] = (T)A[i];
        barrier(L);
    }
    for (int l = last - 1; l >= 0; --l) {
        const TailLv<T>& L = g.lv[l];
        const TailLv<T>& C = g.lv[l + 1];
        if (L.nc == 1 && rank != 0) continue;
        if (!(one && l + 1 == last)) {
            if (L.nc > 1 && C.nc == 1) cl.sync();  // the first CTA's levels are done
            int z0;
            const int pn = own(L, z0);
            prolong_share<T, FLAT, CH>(L, C, sm + L.ox, sm + C.ox, z0, pn, rank);
            barrier(L);
        }
        smooth_level(L, L.nu2, false);
    }
    {
        const TailLv<T>& L = g.lv[0];
        int z0;
        const int pn = own(L, z0), total = pn * L.nx * L.ny;
        T* gx = g.gx + (size_t)z0 * L.nx * L.ny;
        for (int i = threadIdx.x; i < total; i += blockDim.x) gx[i] = sm[L.ox + i];
    }
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

template <typename T>
const void* tail_kernel(bool flat, bool channel) {
    if (flat) return (const void*)k_mg_tail<T, true, false>;
    return channel ? (const void*)k_mg_tail<T, false, true> : (const void*)k_mg_tail<T, false, false>;
}

// the kernels' opt-ins on the current device; false where it refuses clusters of 16
bool tail_attributes() {
    bool ok16 = true;
    for (const void* f : {tail_kernel<float>(true, false), tail_kernel<float>(false, false),
                          tail_kernel<float>(false, true), tail_kernel<double>(true, false),
                          tail_kernel<double>(false, false), tail_kernel<double>(false, true)}) {
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem);
        if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ok16 = false;
    }
    cudaGetLastError();
    return ok16;
}

// CTAs per cluster: 16 where the device takes a non-portable size, else 8, else 1
int tail_cluster() {
    static const int cs = [] {
        const bool ok16 = tail_attributes();
        for (int c : {16, 8}) {
            if (c == 16 && !ok16) continue;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(kTailThreads);
            cfg.dynamicSmemBytes = kTailSmem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, tail_kernel<double>(false, true), &cfg) == cudaSuccess && n > 0)
                return c;
            cudaGetLastError();
        }
        return 1;
    }();
    return cs;
}

// Largest level of the tail by element size. FP32: a 32^3 level takes 15 us in
// the cluster and 16 us in its nine level launches, and its launches go.
// FP64: a 32^3 level takes 48 us on 16 SMs' FP64 pipes and 33 us in launches
// over all of them, a 128^2 one 19 us against 28.
constexpr long long tail_cells(size_t elem) { return elem == sizeof(float) ? kTailCells : kTailCells / 2; }

// Slabs and shared-memory offsets of the levels; bytes per CTA, 0 where the
// tail cannot take them
template <typename T>
size_t tail_layout(const TailLevels<T>& a, int cs, TailArgs<T>* g) {
    size_t off = 0;  // in T
    for (int l = 0; l < a.nlev; ++l) {
        const Dims& d = a.d[l];
        TailLv<T>& L = g->lv[l];
        const bool flat = d.nz == 1 && a.flat;
        L.nx = d.nx;
        L.ny = flat ? 1 : d.ny;
        L.nz = flat ? d.ny : d.nz;
        const long long cells = d.ncell();
        if (cells > (a.nlev == 1 ? kTailCells : tail_cells(sizeof(T))) || L.nz < 1) return 0;
        // FP64: one SM's FP64 pipe (two lanes per clock) makes sharing pay from 128
        // cells; FP32 levels of up to 512 cells are faster behind block barriers
        const int local = sizeof(T) == sizeof(double) ? 128 : 512;
        const bool alone = cs == 1 || cells <= local;
        L.P = alone ? L.nz : (L.nz + cs - 1) / cs;
        if (!alone && L.P > 1 && (L.P & 1)) ++L.P;  // fine planes in coarse pairs
        L.nc = (L.nz + L.P - 1) / L.P;
        L.mP = fdiv_magic(L.P);
        L.mhx = fdiv_magic(d.nx / 2);
        L.mny = fdiv_magic(L.ny);
        L.mcy = fdiv_magic(std::max(1, L.ny / 2));
        L.off = T(d.n) * T(d.n);
        L.inv = T(1) / (T(d.n) * T(d.n));
        const size_t slab = (size_t)L.P * L.nx * L.ny;
        L.ox = (int)off;
        L.ob = (int)(off + slab);
        L.orr = (int)(off + 2 * slab);
        off += (l + 1 < a.nlev ? 3 : 2) * slab;
        off = (off + 3) & ~(size_t)3;
        L.nu1 = a.nu1[l];
        L.nu2 = a.nu2[l];
        L.red = restrict_after_sweep(d, sizeof(T), L.nu1);
        L.black = prolong_before_sweep(d, sizeof(T), L.nu2);
        L.omega = d.nx < kOmegaMinNx ? T(1) : T(a.omega);
        if (l + 1 < a.nlev && (d.nx & 1)) return 0;
    }
    const TailLv<T>& L = g->lv[a.nlev - 1];
    const size_t slab = (size_t)L.P * L.nx * L.ny;
    size_t dbl = (off * sizeof(T) + 15) / 16 * 2;
    g->ofa = (int)dbl;
    g->ofb = (int)(dbl + slab);
    return (dbl + 2 * slab) * sizeof(double);
}

}  // namespace

template <typename T>
bool vcycle_tail_ok(const TailLevels<T>& a) {
    if (a.nlev < 1 || a.nlev > kMaxTailLevels || !a.basis.vx) return false;
    TailArgs<T> g{};
    const int cs = tail_cluster();
    const size_t bytes = tail_layout(a, cs, &g);
    return bytes > 0 && bytes <= kTailSmem;
}

template <typename T>
void launch_vcycle_tail(const TailLevels<T>& a, cudaStream_t s) {
    TailArgs<T> g{};
    int cs = tail_cluster();
    size_t bytes = tail_layout(a, cs, &g);
    // one CTA where every level is the first CTA's own
    if (g.lv[0].nc == 1) cs = 1;
    g.nlev = a.nlev;
    g.flat = a.flat;
    g.channel = a.d[0].channel;
    g.x_zero = a.x_zero;
    g.gx = a.x;
    g.gb = a.b;
    g.vx = a.basis.vx;
    g.vy = a.basis.vy;
    g.vz = a.basis.vz;
    g.lx = a.basis.lx;
    g.ly = a.basis.ly;
    g.lz = a.basis.lz;
    g.n2 = (double)a.d[a.nlev - 1].n * (double)a.d[a.nlev - 1].n;
    g.status = a.status;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // errors reach the caller's cudaGetLastError
    if (a.flat) cudaLaunchKernelEx(&cfg, k_mg_tail<T, true, false>, g);
    else if (g.channel) cudaLaunchKernelEx(&cfg, k_mg_tail<T, false, true>, g);
    else cudaLaunchKernelEx(&cfg, k_mg_tail<T, false, false>, g);
}

void vcycle_tail_attributes() { tail_attributes(); }

template bool vcycle_tail_ok<float>(const TailLevels<float>&);
template bool vcycle_tail_ok<double>(const TailLevels<double>&);
template void launch_vcycle_tail<float>(const TailLevels<float>&, cudaStream_t);
template void launch_vcycle_tail<double>(const TailLevels<double>&, cudaStream_t);

}  // namespace afmib
