// Multigrid tail: the V-cycle below a level of at most kTailCells cells (32^3,
// or a 2D grid of 128 x 256 cells) in one launch on one thread-block cluster.
//
// The coarse levels are a few thousand cells, so a launch per phase costs more
// than the phase, and one block is bound by the shared-memory latency of its
// 45 phases in FP32 and by one SM's FP64 pipe in FP64. Here a cluster of up to
// 16 CTAs holds every level in distributed shared memory: a CTA owns a slab of
// z planes (rows of y on a 2D grid) of each level and reads the neighbouring
// slabs' planes through the cluster's shared-memory window; the levels too small
// to share stay in the first CTA. The coarsest level is solved directly in FP64 in
// the tensor-product eigenbasis of its Laplacian (six short dense transforms; by its
// inverse matrix on up to kDirectCells cells), with the constant mode dropped: what
// the mean removal and CG of src/mg/solver.h:264-271 converge to.
//
// Every cell takes the level kernels' expressions with the same terms in the
// same order (lap_row2, k_rbgs_first, restrict_cell2, prolong_cell2 of
// kernels_mg.cu), so the V-cycle equals the launch-by-launch one bit for bit.
//
// The phases are bound by latency (measured, in clocks: a cluster barrier 480 idle
// and 1100 to 1700 between phases, a load from another CTA's shared memory 255 and
// 11 to 19 per warp of them, local 51, a dependent FP64 instruction 64, and one SM
// issues an FP64 warp instruction every 16 to 19), so: a thread keeps its cells and
// right-hand sides in registers for all phases of a level; a sweep from zero takes
// one phase in FP32; the restriction sums each fine plane in the CTA that holds it
// and moves four sums per coarse cell instead of 32 or 64 taps; the prolongation
// copies the coarse planes it reads.
// Kernel text counts too: every phase runs a few times per launch and its first
// pass waits for its instructions (a variant for two blocks per thread in registers
// took the 32^3 level's colours from 1000 to 1700 clocks).
//
// Measured on GB300 (us per launch, launches back to back; about 5 more inside a
// V-cycle, where its instructions are cold): FP32 from 32^3 21.8 (38.6 with a phase
// per half sweep, cells decoded in every phase, all taps moved between CTAs and levels
// down to one cell; 56 with the 32^3 level in launches of its own and one block below
// it), FP64 from 16^3 20.9 (41.0; 121 in one block), FP64 2D from 128^2 39.4 (63.5),
// FP32 from 24x20x28 to 6x5x7 20.9 (28.7), a coarsest 15^3 level with the 30^3 above
// it 31.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "kernels.h"
#include "mg_cells.cuh"

namespace cg = cooperative_groups;

namespace afmib {

namespace {

constexpr int kTailThreads = 512;  // at most
constexpr size_t kTailSmem = 200 * 1024;

// One level of the tail. On a 2D grid the slabs are rows: ny = 1 and nz is the
// grid's y extent (flat).
template <typename T>
struct TailLv {
    int nx, ny, nz;
    int P, nc;                        // planes per CTA (1, even, or all), CTAs that own any
    unsigned mP, mhx, mny, mcy;       // division by P, nx/2, ny and ny/2 (fdiv)
    int ox, ob, orr, os;              // offsets of x, b, r and the transfer planes in every CTA's shared memory, in T
    int nu1, nu2, red, black;         // restrict_after_sweep, prolong_before_sweep
    T omega, inv, off;                // off = n^2 and inv = 1 / n^2, as the level kernels round them
};
template <typename T>
struct TailArgs {
    TailLv<T> lv[kMaxTailLevels];
    int nlev, flat, channel, x_zero;
    int cells;     // of the coarsest level
    int ofa, ofb;  // the coarsest solve's two FP64 vectors, in doubles
    int ofg;       // its inverse, where that is at hand (0: not)
    T* gx;
    const T* gb;
    const double* inverse;
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
// (ldr: free to move, for a phase that writes elsewhere and has no barrier in it)
__device__ __forceinline__ float ldr(unsigned a, float) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ double ldr(unsigned a, double) {
    double v;
    asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
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

// the same by rank
template <typename T>
__device__ __forceinline__ T ld_at(unsigned a, int own, int rank) {
    return own == rank ? lds(a, T(0)) : ldc(mapa(a, own), T(0));
}

// The cells of a thread: the pair x = 2t, 2t + 1 of a row on ZB planes, two red
// and two black cells (one each for ZB 1), and what lies around them, in elements
// of the CTA's slab from its first one. Between them the cells are in registers;
// a cell reads one neighbour beyond the pair along x, two along y and one along z.
struct Block {
    int a;         // cell 2t of the first plane
    int xl, xr;    // from a: the cells left of 2t and right of 2t + 1
    int yl, yh;    // from a cell: its neighbours in y (unused beyond a channel wall)
    int zl, zh;    // cell 2t of the planes below and above, in their CTA's slab
    int ol, oh;    // the CTAs they belong to
    int y, p;      // p: the red cell of the first plane is 2t + p
};
template <typename T, bool FLAT, int ZB>
__device__ __forceinline__ Block block_of(const TailLv<T>& L, int z0, int rank, int t, int zb, int y) {
    const int nx = L.nx, ny = L.ny, sxy = nx * ny, zl = zb * ZB, z = z0 + zl;
    Block q;
    q.a = nx * (y + ny * zl) + 2 * t;
    q.xl = t == 0 ? nx - 1 : -1;
    q.xr = 2 * t + 2 == nx ? 2 - nx : 2;
    q.yl = y > 0 ? -nx : sxy - nx;
    q.yh = y < ny - 1 ? nx : nx - sxy;
    const int zm = z == 0 ? L.nz - 1 : z - 1, zp = z + ZB >= L.nz ? 0 : z + ZB;
    auto own = [&](int zz) { return L.nc == 1 ? 0 : fdiv(zz, L.mP); };
    q.ol = own(zm);
    q.oh = own(zp);
    q.zl = q.a + sxy * (zm - q.ol * L.P - zl);
    q.zh = q.a + sxy * (zp - q.oh * L.P - zl);
    if (L.nc == 1) q.ol = q.oh = rank;
    q.y = y;
    q.p = (y + z) & 1;
    return q;
}

// The nu sweeps of a level and, with res, the residual r = b - L x after them, on a
// block per thread in registers, or pass by pass on larger slabs (first: the sweeps
// start from x = 0, whatever x holds). Each phase begins with a wait for what it
// reads and none ends with one.
// (Functions of their own, not inlined at their call sites: the kernel runs each a
// few times on one block per SM, and inlined copies spilled registers and missed
// the instruction cache.)
template <typename T, bool FLAT, bool CH, bool DIST, int ZB>
__device__ __noinline__ void smooth(const TailLv<T>& L, unsigned x0, int z0, int pn, int rank, int nu, bool first,
                                    bool res) {
    auto wait = [&]() {
        if constexpr (DIST) cg::this_cluster().sync();
        else __syncthreads();
    };
    constexpr unsigned sz = sizeof(T);
    const int hx = L.nx >> 1, ny = L.ny, total = pn / ZB * ny * hx, bd = blockDim.x, tid = threadIdx.x;
    const unsigned db = sz * (unsigned)(L.ob - L.ox), dr = sz * (unsigned)(L.orr - L.ox), ps = sz * (unsigned)(L.nx * ny);
    const T inv = L.inv, omega = L.omega, off = L.off;
    const bool red_only = L.red;
    // a block as addresses (zl, zh: bit 0 set in another CTA's window)
    struct Addr {
        unsigned a, zl, zh;
        int xl, xr, yl, yh, y, p;
    };
    auto decode = [&](int e) {
        const int row = fdiv(e, L.mhx), t = e - row * hx;
        const int zb = FLAT ? row : fdiv(row, L.mny), y = FLAT ? 0 : row - zb * ny;
        const Block q = block_of<T, FLAT, ZB>(L, z0, rank, t, zb, y);
        Addr r;
        r.a = x0 + sz * q.a;
        r.xl = (int)sz * q.xl;
        r.xr = (int)sz * q.xr;
        r.yl = (int)sz * q.yl;
        r.yh = (int)sz * q.yh;
        const unsigned zl = x0 + sz * q.zl, zh = x0 + sz * q.zh;
        r.zl = !DIST || q.ol == rank ? zl : mapa(zl, q.ol) | 1u;
        r.zh = !DIST || q.oh == rank ? zh : mapa(zh, q.oh) | 1u;
        r.y = q.y;
        r.p = q.p;
        return r;
    };
    auto ldz = [&](unsigned a) { return DIST && (a & 1u) ? ldc(a & ~1u, T(0)) : lds(a, T(0)); };
    auto count = [&](int y) { return FLAT ? 4 : (CH ? 6 - (y == 0) - (y == ny - 1) : 6); };
    auto relax = [&](T S, T b, T old, int c) {
        const T rc = FLAT || (CH && c == 4) ? T(0.25) : (CH && c == 5 ? T(1.0 / 5.0) : T(1.0 / 6.0));
        T v = gs_value(S, b, inv, rc);
        return over_relaxed(v, old, omega);
    };
    // neighbour sum of cell s of plane k: lap_row2's terms in its order; get(address,
    // y) reads a cell outside the block, getz one of the planes beside the block
    auto sum = [&](const Addr& q, const T (&v)[ZB][2], int k, int s, auto get, auto getz) {
        const unsigned a = q.a + k * ps, c = a + s * sz;
        const T xi = s ? v[k][0] : v[k][1], xo = get(a + (s ? q.xr : q.xl), q.y);
        const T lo = k == 0 ? getz(q.zl + s * sz) : (s ? v[0][1] : v[0][0]);
        const T hi = k == ZB - 1 ? getz(q.zh + s * sz) : (s ? v[ZB - 1][1] : v[ZB - 1][0]);
        T S = (xi + xo) + (lo + hi);
        if (!FLAT) {
            if (CH) {
                if (q.y > 0) S += get(c + q.yl, q.y - 1);
                if (q.y < ny - 1) S += get(c + q.yh, q.y + 1);
            } else {
                S += get(c + q.yl, 0) + get(c + q.yh, 0);
            }
        }
        return S;
    };
    auto plain = [&](unsigned a, int) { return lds(a, T(0)); };
    auto load = [&](const Addr& q, T (&x)[ZB][2], T (&b)[ZB][2], bool wx) {
#pragma unroll
        for (int k = 0; k < ZB; ++k)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                b[k][s] = lds(q.a + k * ps + s * sz + db, T(0));
                if (wx) x[k][s] = lds(q.a + k * ps + s * sz, T(0));
            }
    };
    // one colour of a block; its reads of shared memory precede its writes
    auto colour = [&](const Addr& q, T (&x)[ZB][2], const T (&b)[ZB][2], int col) {
        T v[ZB];
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k ^ col;
            v[k] = relax(sum(q, x, k, s, plain, ldz), s ? b[k][1] : b[k][0], s ? x[k][1] : x[k][0], count(q.y));
        }
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k ^ col;
            x[k][0] = s ? x[k][0] : v[k];
            x[k][1] = s ? v[k] : x[k][1];
            sts(q.a + k * ps + s * sz, v[k]);
        }
    };
    // the reds from x = 0 (their sums are zero), the blacks cleared
    auto red0 = [&](const Addr& q, T (&x)[ZB][2], const T (&b)[ZB][2]) {
        const T z = T(0);
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k;
            const T v = relax(z, s ? b[k][1] : b[k][0], z, count(q.y));
            x[k][0] = s ? z : v;
            x[k][1] = s ? v : z;
            sts(q.a + k * ps, x[k][0]);
            sts(q.a + k * ps + sz, x[k][1]);
        }
    };
    // both colours from x = 0: the reds around a black cell are formed from b. Not
    // in FP64, where a black cell's extra operations take longer (1300 clocks) than
    // the barrier that they save.
    constexpr bool kFuse = sizeof(T) == sizeof(float);
    auto sweep0 = [&](const Addr& q, T (&x)[ZB][2], const T (&b)[ZB][2]) {
        const T z = T(0);
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k;
            const T v = relax(z, s ? b[k][1] : b[k][0], z, count(q.y));
            x[k][0] = s ? z : v;
            x[k][1] = s ? v : z;
        }
        auto red = [&](unsigned a, int y) { return relax(z, lds(a + db, z), z, count(y)); };
        auto redz = [&](unsigned a) { return relax(z, ldz(a + db), z, count(q.y)); };
        T v[ZB];
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k ^ 1;
            v[k] = relax(sum(q, x, k, s, red, redz), s ? b[k][1] : b[k][0], z, count(q.y));
        }
#pragma unroll
        for (int k = 0; k < ZB; ++k) {
            const int s = q.p ^ k ^ 1;
            x[k][0] = s ? x[k][0] : v[k];
            x[k][1] = s ? v[k] : x[k][1];
            sts(q.a + k * ps, x[k][0]);
            sts(q.a + k * ps + sz, x[k][1]);
        }
    };
    auto resid = [&](const Addr& q, const T (&x)[ZB][2], const T (&b)[ZB][2]) {
        const int c = count(q.y);
        const T cc = FLAT || (CH && c == 4) ? T(4) : (CH && c == 5 ? T(5) : T(6));
#pragma unroll
        for (int k = 0; k < ZB; ++k)
#pragma unroll
            for (int col = 0; col < 2; ++col) {
                if (col == 1 && red_only) continue;  // plane_sums does not read the black cells
                const int s = q.p ^ k ^ col;
                const T r = (s ? b[k][1] : b[k][0]) - off * (sum(q, x, k, s, plain, ldz) - cc * (s ? x[k][1] : x[k][0]));
                sts(q.a + k * ps + s * sz + dr, r);
            }
    };
    // by level, not by the CTA's own share: every CTA of the cluster takes the same barriers
    if (L.P / ZB * ny * hx <= bd) {
        Addr q;
        T x[ZB][2], b[ZB][2];
        const bool any = tid < total;
        if constexpr (DIST) cg::this_cluster().barrier_arrive();
        if (any) q = decode(tid);
        if constexpr (DIST) cg::this_cluster().barrier_wait();
        else __syncthreads();
        if (any) load(q, x, b, !first);
        int j = 0;
        if (first) {
            j = kFuse ? 2 : 1;
            if (any) {
                if (kFuse) sweep0(q, x, b);
                else red0(q, x, b);
            }
        }
        for (; j < 2 * nu; ++j) {
            if (j > 0) wait();
            if (any) colour(q, x, b, j & 1);
        }
        if (res) {
            wait();
            if (any) resid(q, x, b);
        }
        return;
    }
    auto pass = [&](bool wx, auto f) {
        wait();
        for (int e = tid; e < total; e += bd) {
            const Addr q = decode(e);
            T x[ZB][2], b[ZB][2];
            load(q, x, b, wx);
            f(q, x, b);
        }
    };
    if (first && kFuse) pass(false, [&](const Addr& q, T (&x)[ZB][2], T (&b)[ZB][2]) { sweep0(q, x, b); });
    else if (first) pass(false, [&](const Addr& q, T (&x)[ZB][2], T (&b)[ZB][2]) { red0(q, x, b); });
    for (int j = first ? 2 - !kFuse : 0; j < 2 * nu; ++j)
        pass(true, [&](const Addr& q, T (&x)[ZB][2], T (&b)[ZB][2]) { colour(q, x, b, j & 1); });
    if (res) pass(true, [&](const Addr& q, T (&x)[ZB][2], T (&b)[ZB][2]) { resid(q, x, b); });
}

// Restriction, first part: the (1,3,3,1)^2-weighted sums of the CTA's own fine
// planes (rows on a 2D grid) at every coarse (xc, yc): restrict_taps' and
// restrict_rows' plane sums
template <typename T, bool FLAT, bool CH>
__device__ __noinline__ void plane_sums(const TailLv<T>& L, unsigned r0, unsigned s0, int z0, int pn) {
    constexpr unsigned sz = sizeof(T);
    const int nx = L.nx, ny = L.ny, hx = nx >> 1, cy = FLAT ? 1 : ny >> 1, total = pn * hx * cy;
    const unsigned mhx = L.mhx, mcy = L.mcy;
    const bool red = L.red;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int row = fdiv(e, mhx), xc = e - row * hx;
        const int zl = FLAT ? row : fdiv(row, mcy), yc = FLAT ? 0 : row - zl * cy;
        const unsigned r = r0 + sz * (unsigned)(zl * nx * ny);
        const int xs[4] = {xc == 0 ? nx - 1 : 2 * xc - 1, 2 * xc, 2 * xc + 1, 2 * xc + 2 == nx ? 0 : 2 * xc + 2};
        auto rowsum = [&](int y) {
            const unsigned a = r + sz * (unsigned)(nx * y);
            auto get = [&](int x) { return ldr(a + sz * (unsigned)x, T(0)); };
            const bool odd = ((y + z0 + zl) & 1) != 0;  // red_row's taps
            if (red) return fma_t(T(3), get(odd ? xs[2] : xs[1]), get(odd ? xs[0] : xs[3]));
            return full4<T>(get(xs[0]), get(xs[1]), get(xs[2]), get(xs[3]));
        };
        T acc;
        if (FLAT) {
            acc = rowsum(0);
        } else {
            const int y0 = yc == 0 ? (CH ? 0 : ny - 1) : 2 * yc - 1, y3 = 2 * yc + 2 == ny ? (CH ? ny - 1 : 0) : 2 * yc + 2;
            acc = full4<T>(rowsum(y0), rowsum(2 * yc), rowsum(2 * yc + 1), rowsum(y3));
        }
        sts(s0 + sz * (unsigned)e, acc);
    }
}
// second part, by the CTA that owns the coarse plane: b of C from four planes' sums
template <typename T, bool FLAT>
__device__ __noinline__ void restrict_pull(const TailLv<T>& L, const TailLv<T>& C, unsigned s0, unsigned cb, int z0c,
                                           int pnc, int rank) {
    constexpr unsigned sz = sizeof(T);
    const int cxy = C.nx * C.ny, nz = L.nz, total = pnc * cxy;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int row = fdiv(e, L.mhx), zl = FLAT ? row : fdiv(row, L.mcy), p = e - zl * cxy, zc = z0c + zl;
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int zz = 2 * zc - 1 + k, z = zz < 0 ? nz - 1 : (zz >= nz ? zz - nz : zz);
            const int own = L.nc == 1 ? rank : fdiv(z, L.mP);
            const unsigned a = s0 + sz * (unsigned)(p + cxy * (z - (L.nc == 1 ? 0 : own * L.P)));
            v[k] = ld_at<T>(a, own, rank);
        }
        sts(cb + sz * (unsigned)e, full4<T>(v[0], v[1], v[2], v[3]) * T(FLAT ? 1.0 / 64.0 : 1.0 / 512.0));
    }
}

// The coarse planes that the CTA's share of the prolongation reads, copied from
// the CTAs that own them: from plane (z0 - 1) >> 1 (-1: the last one) on
template <typename T, bool FLAT>
__device__ __noinline__ void prolong_copy(const TailLv<T>& L, const TailLv<T>& C, unsigned cx, unsigned stage, int z0,
                                          int pn, int rank) {
    if (pn == 0) return;
    constexpr unsigned sz = sizeof(T);
    const int cxy = C.nx * C.ny, first = (z0 - 1) >> 1, total = (((z0 + pn - 2) >> 1) + 2 - first) * cxy;
    const unsigned mhx = L.mhx, mcy = L.mcy, mP = C.mP;
    const int cP = C.P, cz = C.nz;
    const bool shared = C.nc > 1;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int row = fdiv(e, mhx), j = FLAT ? row : fdiv(row, mcy), p = e - j * cxy;
        const int zz = first + j, z = zz < 0 ? cz - 1 : (zz >= cz ? zz - cz : zz);
        const int own = shared ? fdiv(z, mP) : 0;
        sts(stage + sz * (unsigned)e, ld_at<T>(cx + sz * (unsigned)(p + cxy * (z - own * cP)), own, rank));
    }
}

// x += P xc on the CTA's planes: fine plane z = 2 zc + 1 is the first (nearest
// to zc) and 2 zc + 2 the second (nearest to zc + 1) of a coarse pair; cx: the
// whole coarse level or (DIST) prolong_copy's planes
template <typename T, bool FLAT, bool CH, bool DIST>
__device__ __noinline__ void prolong_share(const TailLv<T>& L, const TailLv<T>& C, unsigned X, unsigned cx, int z0,
                                           int pn) {
    constexpr unsigned sz = sizeof(T);
    const int nx = L.nx, ny = L.ny, sxy = nx * ny, hx = C.nx, cy = C.ny, cxy = hx * cy, cz = C.nz, total = pn * hx * cy;
    const unsigned mhx = L.mhx, mcy = L.mcy;
    const bool black = L.black;
    const int first = (z0 - 1) >> 1;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int row = fdiv(e, mhx), xc = e - row * hx;
        const int zl = FLAT ? row : fdiv(row, mcy), yc = FLAT ? 0 : row - zl * cy;
        const int z = z0 + zl, zc = (z - 1) >> 1;
        const int p = DIST ? zc - first : (zc < 0 ? cz - 1 : zc), q = DIST ? p + 1 : (zc + 1 == cz ? 0 : zc + 1);
        const int a = hx * yc, b = yc + 1 == cy ? 0 : a + hx;
        const unsigned near = cx + sz * (unsigned)(cxy * ((z & 1) ? p : q)), far = cx + sz * (unsigned)(cxy * ((z & 1) ? q : p));
        const int xn = xc + 1 == hx ? 0 : xc + 1;
        const int xf[2] = {2 * xc + 1, 2 * xc + 2 == nx ? 0 : 2 * xc + 2};
        const unsigned Xp = X + sz * (unsigned)(zl * sxy);
        auto at = [&](unsigned plane, int i) { return ldr(plane + sz * (unsigned)i, T(0)); };
        auto put = [&](int x, int y, T v, T s) {
            const unsigned i = Xp + sz * (unsigned)(x + nx * y);
            sts(i, fma_t(v, s, ldr(i, T(0))));  // no other thread's or iteration's cell
        };
        const int rz = (z & 1) ? 0 : 1;  // on a 2D grid z is y
        const T nl = at(near, xc + a), nr = at(near, xn + a), fl = at(far, xc + a), fr = at(far, xn + a);
        if (FLAT) {
            prolong_row2(nl, nr, fl, fr, black_col(black, rz, 1), [&](int rx, T v, T s) { put(xf[rx], 0, v, s); });
            continue;
        }
        if (!CH || yc < cy - 1) {
            const int yf[2] = {2 * yc + 1, 2 * yc + 2 == ny ? 0 : 2 * yc + 2};
            prolong_plane4(nl, nr, at(near, xc + b), at(near, xn + b), fl, fr, at(far, xc + b), at(far, xn + b), black, rz,
                           [&](int rx, int ry, T v, T s) { put(xf[rx], yf[ry], v, s); });
        }
        if (CH && yc == 0)
            prolong_row2(nl, nr, fl, fr, black_col(black, 1, rz), [&](int rx, T v, T s) { put(xf[rx], 0, v, s); });
        if (CH && yc == cy - 1)
            prolong_row2(nl, nr, fl, fr, black_col(black, 0, rz), [&](int rx, T v, T s) { put(xf[rx], ny - 1, v, s); });
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
    constexpr int kWords = (int)(sizeof(g) / sizeof(int));
    for (int i = threadIdx.x; i < kWords; i += blockDim.x)
        reinterpret_cast<int*>(&g)[i] = reinterpret_cast<const int*>(&args)[i];
    const cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    if (args.ofg && rank == 0) {  // arrives while the levels above are smoothed
        const int n = args.cells * args.cells / 2;
        const unsigned to = (unsigned)__cvta_generic_to_shared(tsm) + 8u * (unsigned)args.ofg;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * i), "l"(args.inverse + 2 * i) : "memory");
    }
    auto own = [&](const TailLv<T>& L, int& z0) {
        z0 = rank * L.P;
        const int n = L.nz - z0;
        return rank >= L.nc ? 0 : (n < L.P ? n : L.P);
    };
    auto barrier = [&](const TailLv<T>& L) {
        if (L.nc > 1) cl.sync();
        else __syncthreads();
    };
    wait_launch();
    {
        const TailLv<T>& L = args.lv[0];
        int z0;
        const int pn = own(L, z0), total = pn * L.nx * L.ny;
        const T* gb = args.gb + (size_t)z0 * L.nx * L.ny;
        const T* gx = args.gx + (size_t)z0 * L.nx * L.ny;
        for (int i = threadIdx.x; i < total; i += 4 * blockDim.x) {  // four loads in flight per array
            T vb[4], vx[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = i + k * blockDim.x;
                vb[k] = j < total ? gb[j] : T(0);
                vx[k] = j < total && !args.x_zero ? gx[j] : T(0);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = i + k * blockDim.x;
                if (j < total) {
                    sm[L.ob + j] = vb[k];
                    if (!args.x_zero) sm[L.ox + j] = vx[k];
                }
            }
        }
        __syncthreads();  // the level's first phase waits for the other CTAs
    }
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(sm);
    auto at = [&](int offset) { return sbase + (unsigned)sizeof(T) * (unsigned)offset; };
    auto smooth_level = [&](int l, int nu, bool first, bool res) {
        const TailLv<T>& L = g.lv[l];
        int z0;
        const int pn = own(L, z0);
        if (first && nu < 1) {
            for (int i = threadIdx.x; i < pn * L.nx * L.ny; i += blockDim.x) sm[L.ox + i] = T(0);
            first = false;
        }
        // two planes per block where a thread has two pairs anyway: half the loads
        // along z. Not in FP64, where a warp's instructions take 64 clocks each: a
        // warp with two cells per lane instead of two warps doubles a phase.
        if (L.nc == 1) smooth<T, FLAT, CH, false, 1>(L, at(L.ox), z0, pn, rank, nu, first, res);
        else if (sizeof(T) == sizeof(double) || L.P == 1 || L.P * L.ny * (L.nx >> 1) <= (int)blockDim.x)
            smooth<T, FLAT, CH, true, 1>(L, at(L.ox), z0, pn, rank, nu, first, res);
        else if constexpr (sizeof(T) == sizeof(float))
            smooth<T, FLAT, CH, true, 2>(L, at(L.ox), z0, pn, rank, nu, first, res);
        __syncthreads();
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
        smooth_level(l, L.nu1, l > 0 || g.x_zero, down);
        if (!down) break;
        int z0, z0c;
        const int pn = own(L, z0), pnc = own(C, z0c);
        plane_sums<T, FLAT, CH>(L, at(L.orr), at(L.os), z0, pn);
        barrier(L);
        restrict_pull<T, FLAT>(L, C, at(L.os), at(C.ob), z0c, pnc, rank);
    }
    __syncthreads();
    // coarsest level: V^T diag(1 / lambda) V b over the three axes, the
    // constant mode dropped; rows of fixed-order FP64 sums
    if (one) {
        if (last == 0 && rank == 0 && threadIdx.x == 0) sm[g.lv[0].ox] = T(0);
        if (last == 0) __syncthreads();
    } else if (g.ofg) {
        // x = G b, by rows of the symmetric G: a warp takes 32 cells and a share of
        // the terms (the same shares whatever the block), added in order
        if (rank == 0) {
            const TailLv<T>& L = g.lv[last];
            const int n = g.cells, groups = (n + 31) >> 5, parts = 8 / groups, w = threadIdx.x >> 5;
            const int i = (w % groups) * 32 + (threadIdx.x & 31), part = w / groups;
            const int j0 = part * n / parts, j1 = (part + 1) * n / parts;
            const double* G = (const double*)tsm + g.ofg;
            double *sums = (double*)tsm + g.ofa, *B = (double*)tsm + g.ofb;
            if (threadIdx.x < n) B[threadIdx.x] = (double)sm[L.ob + threadIdx.x];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (i < n && part < parts) {
                double s = 0.0;
#pragma unroll 4
                for (int j = j0; j < j1; ++j) s += G[j * n + i] * B[j];
                sums[part * n + i] = s;
            }
            __syncthreads();
            if (threadIdx.x < n) {
                double s = sums[threadIdx.x];
                for (int k = 1; k < parts; ++k) s += sums[k * n + threadIdx.x];
                if (!isfinite(s)) atomicExch(g.status, 3);
                sm[L.ox + threadIdx.x] = (T)s;
            }
            __syncthreads();
        }
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
            barrier(L);  // the coarse level is done, wherever it is
            int z0;
            const int pn = own(L, z0);
            const unsigned X = at(L.ox), cx = at(C.ox), stage = at(L.os);
            if (L.nc > 1) {
                prolong_copy<T, FLAT>(L, C, cx, stage, z0, pn, rank);
                __syncthreads();
                prolong_share<T, FLAT, CH, true>(L, C, X, stage, z0, pn);
            } else {
                prolong_share<T, FLAT, CH, false>(L, C, X, cx, z0, pn);
            }
        }
        smooth_level(l, L.nu2, false, false);
    }
    cl.barrier_arrive();  // no CTA leaves while another may still read its shared memory
    {
        const TailLv<T>& L = g.lv[0];
        int z0;
        const int pn = own(L, z0), total = pn * L.nx * L.ny;
        T* gx = g.gx + (size_t)z0 * L.nx * L.ny;
        for (int i = threadIdx.x; i < total; i += blockDim.x) gx[i] = sm[L.ox + i];
    }
    cl.barrier_wait();
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

// whether a cluster of c CTAs with the tail's shared memory fits the current device
bool cluster_fits(int c) {
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
    if (cudaOccupancyMaxActiveClusters(&n, tail_kernel<double>(false, true), &cfg) == cudaSuccess && n > 0) return true;
    cudaGetLastError();
    return false;
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
        off += 2 * slab;
        if (l + 1 < a.nlev) {
            const size_t cxy = (size_t)(L.nx / 2) * std::max(1, L.ny / 2);
            off += slab;
            L.os = (int)off;
            off += std::max(L.P, L.P / 2 + 2) * cxy;  // plane sums, or the coarse planes of the prolongation
        }
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
    g->cells = (int)a.d[a.nlev - 1].ncell();
    g->inverse = a.basis.inverse;
    g->ofg = 0;
    if (a.basis.inverse && g->cells > 1 && L.nc == 1) {
        g->ofb = (int)(dbl + 8 * (size_t)g->cells);  // after the warps' partial sums
        dbl += 9 * (size_t)g->cells;
        dbl += dbl & 1;
        g->ofg = (int)dbl;
        return (dbl + (size_t)g->cells * g->cells) * sizeof(double);
    }
    return (dbl + 2 * slab) * sizeof(double);
}

}  // namespace

template <typename T>
bool vcycle_tail_ok(const TailLevels<T>& a) {
    if (a.nlev < 1 || a.nlev > kMaxTailLevels || !a.basis.vx) return false;
    TailArgs<T> g{};
    const size_t bytes = tail_layout(a, a.cluster, &g);
    return bytes > 0 && bytes <= kTailSmem;
}

template <typename T>
void launch_vcycle_tail(const TailLevels<T>& a, cudaStream_t s) {
    TailArgs<T> g{};
    int cs = a.cluster;
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
    // a thread per pair of cells of a plane (two planes in FP32) where 512 reach;
    // half of them are faster where that is enough (idle warps cost at barriers)
    int most = 0;
    for (int l = 0; l + 1 < g.nlev; ++l)
        most = std::max(most, g.lv[l].P * g.lv[l].ny * (g.lv[l].nx / 2));
    cfg.blockDim = dim3(most > kTailThreads / 2 ? kTailThreads : kTailThreads / 2);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // launch_dep
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    // errors reach the caller's cudaGetLastError
    if (a.flat) cudaLaunchKernelEx(&cfg, k_mg_tail<T, true, false>, g);
    else if (g.channel) cudaLaunchKernelEx(&cfg, k_mg_tail<T, false, true>, g);
    else cudaLaunchKernelEx(&cfg, k_mg_tail<T, false, false>, g);
}

int vcycle_tail_cluster(int most) {
    const bool ok16 = tail_attributes();
    for (int c : {16, 8, 4, 2})
        if (c <= most && (c < 16 || ok16) && cluster_fits(c)) return c;
    return 1;
}

template bool vcycle_tail_ok<float>(const TailLevels<float>&);
template bool vcycle_tail_ok<double>(const TailLevels<double>&);
template void launch_vcycle_tail<float>(const TailLevels<float>&, cudaStream_t);
template void launch_vcycle_tail<double>(const TailLevels<double>&, cudaStream_t);

}  // namespace afmib
