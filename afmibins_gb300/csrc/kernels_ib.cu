// Immersed-boundary transfer kernels: springs, marker binning by a stable
// device radix sort, deterministic gather spreading and interpolation.
//
// Reference: ib::grid::interpolate (src/ib/grid.h:68-84) computes both
// directions face by face or marker by marker with the cosine 4-point kernel
//   phi(r) = n/4 (1 + cos(pi r n / 2)), |r n| <= 2     (src/ib/grid.h:51-55)
// and finds neighbours with a kd-tree (src/dt/kdtree.h). Here the markers are
// binned by cell instead: a key (tile, cell in tile) per marker is sorted with
// a stable LSD radix sort, so the markers of every cell are contiguous and in
// index order. Spreading then runs one block per output tile of TS^3 cells,
// gathering from the markers binned in the tile's (TS+4)^3 neighbourhood in a
// fixed order: no float atomics, bitwise repeatable.
//
// Weights: for a marker at s = X*n along an axis and faces at j + off, the
// four faces with |j + off - s| < 2 are j = floor(s - off) - 1 + m, m = 0..3,
// and with t = frac(s - off), S = sin(pi t / 2), C = cos(pi t / 2):
//   phi/n = (1 - S)/4, (1 + C)/4, (1 + S)/4, (1 - C)/4      (sum = 1)
// (cos(pi r/2) at r = -1-t, -t, 1-t, 2-t). One sincospi per axis and offset.
#include <algorithm>
#include <type_traits>

#include "dfloat.cuh"
#include "kernels_ib.h"

namespace afmib {

namespace {

__device__ __forceinline__ double sinpi_cospi(double x, double* c) {
    double s;
    sincospi(x, &s, c);
    return s;
}
__device__ __forceinline__ float sinpi_cospi(float x, float* c) {
    float s;
    sincospif(x, &s, c);
    return s;
}

// G_i = k * sum_j (X_j - X_i)
template <typename T>
__global__ void k_springs(int M, const double* __restrict__ X, const int* __restrict__ ns, const int* __restrict__ ni,
                          double k, T* __restrict__ G) {
    wait_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const double xi = X[3 * i], yi = X[3 * i + 1], zi = X[3 * i + 2];
    double sx = 0, sy = 0, sz = 0;
    for (int e = ns[i]; e < ns[i + 1]; ++e) {
        const int j = ni[e];
        sx += X[3 * j] - xi;
        sy += X[3 * j + 1] - yi;
        sz += X[3 * j + 2] - zi;
    }
    G[i] = T(k * sx);
    G[M + i] = T(k * sy);
    G[2 * M + i] = T(k * sz);
}

// Y = L X per marker (L the graph Laplacian of the spring lists), stored
// like X: Y_i = sum_{j in N(i)} (X_j - X_i)
__global__ void k_lap_aos(int M, const double* __restrict__ X, const int* __restrict__ ns, const int* __restrict__ ni,
                          double* __restrict__ Y) {
    wait_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const double xi = X[3 * i], yi = X[3 * i + 1], zi = X[3 * i + 2];
    double sx = 0, sy = 0, sz = 0;
    for (int e = ns[i]; e < ns[i + 1]; ++e) {
        const int j = ni[e];
        sx += X[3 * j] - xi;
        sy += X[3 * j + 1] - yi;
        sz += X[3 * j + 2] - zi;
    }
    Y[3 * i] = sx;
    Y[3 * i + 1] = sy;
    Y[3 * i + 2] = sz;
}

// Springs plus bending from Y = L X: G_i = ks Y_i - kb (L Y)_i. The bending
// term is the force of the discrete energy kb/2 sum_i |(L X)_i|^2 (with
// symmetric lists L is symmetric, so the gradient is kb L L X).
template <typename T>
__global__ void k_spring_bend(int M, const double* __restrict__ Y, const int* __restrict__ ns,
                              const int* __restrict__ ni, double ks, double kb, T* __restrict__ G) {
    wait_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const double yi[3] = {Y[3 * i], Y[3 * i + 1], Y[3 * i + 2]};
    double b[3] = {0, 0, 0};
    for (int e = ns[i]; e < ns[i + 1]; ++e) {
        const int j = ni[e];
        for (int a = 0; a < 3; ++a) b[a] += Y[3 * j + a] - yi[a];
    }
    for (int a = 0; a < 3; ++a) G[(size_t)a * M + i] = T(ks * yi[a] - kb * b[a]);
}

// Per marker: bin key, wrapped cell, and for each axis and offset variant
// (0: faces on integer positions, 1: on half-integers) the base offset
// (first face - cell) and the four weights phi/n.
// DF (FP64 weights only): the sine and cosine by df_sincospi on the FP32
// pipe instead of the FP64 sincospi (the mixed form), weights rounded to FP64
// from their pairs
template <typename T, bool DF>
__global__ void k_marker_prep(Dims d, int TS, int M, const double* __restrict__ X, unsigned* __restrict__ keys,
                              int* __restrict__ vals, MarkerW<T> mw, int* __restrict__ flag) {
    wait_launch();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const int ext[3] = {d.nx, d.ny, d.nz};
    const int TZ = d.nz == 1 ? 1 : TS;  // 2D grids: tiles one cell deep
    int cell[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double s = X[3 * k + a] * d.n;
        const double fs = floor(s);
        cell[a] = wrapi((int)fs, ext[a]);
        if (a == 1 && d.channel && (s < 2.5 || s > d.ny - 2.5)) atomicExch(flag, 1);
        if (!(s == s)) atomicExch(flag, 2);
        if (a == 2 && d.nz == 1) {
            // 2D: the z kernel is the single plane with weight one
            cell[2] = 0;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                mw.dbase[(k * 3 + a) * 2 + v] = 0;
                T* w = mw.w + (((size_t)k * 3 + a) * 2 + v) * 4;
                w[0] = T(1);
                w[1] = w[2] = w[3] = T(0);
            }
            continue;
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const double t = s - 0.5 * v;
            const double ft = floor(t);
            const T frac = T(t - ft);
            mw.dbase[(k * 3 + a) * 2 + v] = (signed char)((int)ft - 1 - (int)fs);
            T* w = mw.w + (((size_t)k * 3 + a) * 2 + v) * 4;
            if constexpr (DF && sizeof(T) == sizeof(double)) {
                df2 hx = df_split(frac);  // frac / 2 exactly
                hx.hi *= 0.5f;
                hx.lo *= 0.5f;
                df2 Sx, Cx;
                df_sincospi(hx, &Sx, &Cx);
                const df2 one = {1.f, 0.f};
                const df2 q[4] = {df_add(one, df_neg(Sx)), df_add(one, Cx), df_add(one, Sx), df_add(one, df_neg(Cx))};
#pragma unroll
                for (int m = 0; m < 4; ++m) w[m] = f32_to_f64(0.25f * q[m].hi) + f32_to_f64(0.25f * q[m].lo);
            } else {
                T C;
                const T S = sinpi_cospi(frac * T(0.5), &C);
                w[0] = T(0.25) * (T(1) - S);
                w[1] = T(0.25) * (T(1) + C);
                w[2] = T(0.25) * (T(1) + S);
                w[3] = T(0.25) * (T(1) - C);
            }
        }
    }
    mw.cell[3 * k] = cell[0];
    mw.cell[3 * k + 1] = cell[1];
    mw.cell[3 * k + 2] = cell[2];
    const int tx = cell[0] / TS, ty = cell[1] / TS, tz = cell[2] / TZ;
    const int ntx = d.nx / TS, nty = d.ny / TS;
    const unsigned tile = (unsigned)(tx + ntx * (ty + nty * tz));
    const unsigned local = (unsigned)((cell[0] % TS) + TS * ((cell[1] % TS) + TS * (cell[2] % TZ)));
    if (keys) keys[k] = tile * (unsigned)(TS * TS * TZ) + local;  // null: weights only
    if (vals) vals[k] = k;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) pairs, 8-bit digits.
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;

__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const unsigned* __restrict__ keys, int n, int shift,
                                                        unsigned* __restrict__ hist, int nblk) {
    wait_launch();
    __shared__ unsigned cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int i = base + r * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nblk + blockIdx.x] = cnt[threadIdx.x];
}

// Exclusive scan of each digit's row hist[digit][nblk], a warp per row; the rows'
// totals go behind them (hist[256 nblk + digit]) and the scatter scans those 256.
// (One block over all of it took 15 us per pass at 200,000 markers and 100 at 10^6.)
__global__ void __launch_bounds__(RS_THREADS) k_rs_scan(unsigned* __restrict__ hist, int nblk) {
    wait_launch();
    const int dig = blockIdx.x * (RS_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    unsigned* row = hist + (size_t)dig * nblk;
    unsigned run = 0;
    for (int i0 = 0; i0 < nblk; i0 += 128) {  // four loads in flight
        unsigned v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i0 + 32 * k + lane < nblk ? row[i0 + 32 * k + lane] : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            unsigned inc = v[k];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            if (i0 + 32 * k + lane < nblk) row[i0 + 32 * k + lane] = run + inc - v[k];
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
    if (lane == 0) hist[(size_t)256 * nblk + dig] = run;
}

// A warp owns RS_ITEMS rows of 32 pairs and counts its digits in a column of its
// own: a pair's position is the digit's start, the blocks before, the warps before,
// the warp's count so far and the rank among the equal digits of the row.
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const unsigned* __restrict__ kin, const int* __restrict__ vin,
                                                           unsigned* __restrict__ kout, int* __restrict__ vout, int n,
                                                           int shift, const unsigned* __restrict__ hist, int nblk) {
    wait_launch();
    constexpr int W = RS_THREADS / 32;
    __shared__ unsigned cnt[256][W + 1];
    __shared__ unsigned wsum[W];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned mine = hist[(size_t)tid * nblk + blockIdx.x], total = hist[(size_t)256 * nblk + tid];
    const int i0 = blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS) + lane;
    unsigned key[RS_ITEMS], rank[RS_ITEMS];
    int val[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const int i = i0 + 32 * r;
        key[r] = i < n ? kin[i] : 0u;
        val[r] = i < n ? vin[i] : 0;
    }
#pragma unroll
    for (int w = 0; w < W; ++w) cnt[tid][w] = 0;
    unsigned inc = total;  // start of digit tid: scan of the totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    unsigned start = inc - total + mine;
    for (int w = 0; w < warp; ++w) start += wsum[w];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const bool valid = i0 + 32 * r < n;
        const unsigned dig = valid ? ((key[r] >> shift) & 255u) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, dig);
        const unsigned before = valid ? cnt[dig][warp] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) cnt[dig][warp] = before + __popc(peers);
        __syncwarp();
        rank[r] = before + __popc(peers & lt);
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const unsigned c = cnt[tid][w];
        cnt[tid][w] = start;
        start += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r)
        if (i0 + 32 * r < n) {
            const unsigned pos = cnt[(key[r] >> shift) & 255u][warp] + rank[r];
            kout[pos] = key[r];
            vout[pos] = val[r];
        }
}

// The same order for up to RS_SMALL pairs in one launch of one block, with the
// tile ranges: the nine launches of three passes and the bins' memsets took 65 us
// at a few thousand markers, launch after launch. The pairs stay in shared memory
// (the values as 16 bits: they are positions); a warp owns a contiguous run of them
// and counts its digits in a column of its own, so that a rank is the warp's count
// so far plus the rank among the equal digits of the row, and the order is stable.
constexpr int RSS_THREADS = 1024, RSS_ITEMS = 8, RS_SMALL = RSS_THREADS * RSS_ITEMS, RSS_COLS = RSS_THREADS / 32 + 1;

// ITEMS rows of 32 pairs per warp
template <int ITEMS>
__global__ void __launch_bounds__(RSS_THREADS, 1) k_sort_small(unsigned* __restrict__ kio, int* __restrict__ vio, int n,
                                                              int bits, int cells_per_tile, int ntiles,
                                                              int* __restrict__ tstart, int* __restrict__ tend,
                                                              int* __restrict__ counts) {
    wait_launch();
    extern __shared__ unsigned rss_smem[];
    unsigned* sk = rss_smem;                           // [ITEMS * RSS_THREADS]
    unsigned* cnt = sk + RSS_THREADS * ITEMS;          // [256][RSS_COLS]
    unsigned* wsum = cnt + 256 * RSS_COLS;             // [32]
    unsigned short* sv = (unsigned short*)(wsum + 32);  // [ITEMS * RSS_THREADS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, i0 = warp * (32 * ITEMS) + lane;
    const unsigned lt = (1u << lane) - 1u;
    for (int t = tid; t < ntiles; t += RSS_THREADS) tstart[t] = tend[t] = 0;
    if (tid < 2) counts[tid] = 0;
    unsigned key[ITEMS], vp[ITEMS];  // vp: value, and position from bit 16
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int i = i0 + 32 * r;
        key[r] = i < n ? kio[i] : 0xffffffffu;  // the padding stays behind equal digits
        vp[r] = i < n ? (unsigned)vio[i] : 0u;
    }
    for (int shift = 0; shift < bits; shift += 8) {
        if (shift > 0) {
#pragma unroll
            for (int r = 0; r < ITEMS; ++r) {
                key[r] = sk[i0 + 32 * r];
                vp[r] = sv[i0 + 32 * r];
            }
        }
        for (int i = tid; i < 256 * RSS_COLS; i += RSS_THREADS) cnt[i] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const unsigned dig = (key[r] >> shift) & 255u, peers = __match_any_sync(0xffffffffu, dig);
            unsigned* c = cnt + dig * RSS_COLS + warp;
            const unsigned before = *c;
            __syncwarp();
            if (lane == __ffs(peers) - 1) *c = before + __popc(peers);
            __syncwarp();
            vp[r] |= (before + __popc(peers & lt)) << 16;
        }
        __syncthreads();
        // exclusive scan by digit, then warp: a thread has eight columns of a digit
        unsigned* c = cnt + (tid >> 2) * RSS_COLS + (tid & 3) * 8;
        unsigned s = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned v = c[k];
            c[k] = s;
            s += v;
        }
        unsigned inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const unsigned w = wsum[lane];
            unsigned x = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned v = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += v;
            }
            wsum[lane] = x - w;
        }
        __syncthreads();
        const unsigned base = wsum[warp] + inc - s;
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] += base;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const unsigned pos = cnt[((key[r] >> shift) & 255u) * RSS_COLS + warp] + (vp[r] >> 16);
            sk[pos] = key[r];
            sv[pos] = (unsigned short)vp[r];
        }
        __syncthreads();
    }
    for (int p = tid; p < n; p += RSS_THREADS) {
        const unsigned k = sk[p], t = k / (unsigned)cells_per_tile;
        kio[p] = k;
        vio[p] = sv[p];
        if (p == 0 || sk[p - 1] / (unsigned)cells_per_tile != t) tstart[t] = p;
        if (p == n - 1 || sk[p + 1] / (unsigned)cells_per_tile != t) tend[t] = p + 1;
    }
}

// tile ranges of the sorted keys: tstart/tend zeroed beforehand
__global__ void k_tile_ranges(const unsigned* __restrict__ keys, int M, int cells_per_tile, int* __restrict__ tstart,
                              int* __restrict__ tend) {
    wait_launch();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const unsigned t = keys[p] / (unsigned)cells_per_tile;
    if (p == 0 || keys[p - 1] / (unsigned)cells_per_tile != t) tstart[t] = p;
    if (p == M - 1 || keys[p + 1] / (unsigned)cells_per_tile != t) tend[t] = p + 1;
}

// Per tile: the slot of each occupied tile (or -1) with its cell-start table
// (ctab[slot][c] = first sorted position of local cell c, c = TS^3 the tile's end,
// by binary search in the tile's sorted key range), and the list of output tiles
// whose (TS+4)^3 neighbourhood holds a marker. Slots are handed out by an atomic
// counter; a slot only names storage, so its value never reaches a result. A block
// takes four tiles at a time: a warp each looks at the neighbours, then all threads
// fill the tables of the occupied ones, searching a copy of the tile's keys (24 us at
// 256^3 cells and 200,000 markers; 28.7 searching global memory).
constexpr int kTileWarps = 4, kTileKeys = 1024;  // keys searched in shared memory
template <int TS, int TZ>
__global__ void __launch_bounds__(32 * kTileWarps) k_tiles(int ntx, int nty, int ntz, int channel,
                                                          const unsigned* __restrict__ keys,
                                                          const int* __restrict__ tstart, const int* __restrict__ tend,
                                                          int* __restrict__ list, int* __restrict__ count,
                                                          int* __restrict__ slot, int* __restrict__ ctab) {
    wait_launch();
    constexpr int C = TS * TS * TZ;
    __shared__ int s_slot[kTileWarps];
    __shared__ unsigned s_key[kTileKeys];
    const int nt = ntx * nty * ntz, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t0 = blockIdx.x * kTileWarps; t0 < nt; t0 += gridDim.x * kTileWarps) {
        const int t = t0 + warp;
        if (t < nt) {
            const int tx = t % ntx, ty = (t / ntx) % nty, tz = t / (ntx * nty);
            bool any = false;
            if (lane < 27) {
                const int yy = ty + lane / 3 % 3 - 1;
                if (!channel || (yy >= 0 && yy < nty)) {
                    const int n = wrapi(tx + lane % 3 - 1, ntx) + ntx * (wrapi(yy, nty) + nty * wrapi(tz + lane / 9 - 1, ntz));
                    any = tend[n] > tstart[n];
                }
            }
            const unsigned vote = __ballot_sync(0xffffffffu, any);
            if (lane == 0) {
                const int sl = (vote >> 13) & 1u ? atomicAdd(count + 1, 1) : -1;  // lane 13: the tile itself
                slot[t] = s_slot[warp] = sl;
                if (vote) list[atomicAdd(count, 1)] = t;
            }
        } else if (lane == 0) {
            s_slot[warp] = -1;
        }
        __syncthreads();
        for (int w = 0; w < kTileWarps; ++w) {
            const int sl = s_slot[w];
            if (sl < 0) continue;
            const int a = tstart[t0 + w], b = tend[t0 + w];
            int* row = ctab + (size_t)sl * (C + 1);
            const bool staged = b - a <= kTileKeys;
            if (staged)
                for (int i = threadIdx.x; i < b - a; i += 32 * kTileWarps) s_key[i] = keys[a + i];
            __syncthreads();
            auto search = [&](auto at) {
                for (int c = threadIdx.x; c <= C; c += 32 * kTileWarps) {
                    const unsigned key = (unsigned)(t0 + w) * C + c;
                    int lo = 0, hi = b - a;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (at(mid) < key) lo = mid + 1; else hi = mid;
                    }
                    row[c] = a + lo;
                }
            };
            if (staged) search([&](int i) { return s_key[i]; });
            else search([&](int i) { return keys[a + i]; });
            __syncthreads();
        }
        __syncthreads();
    }
}

// Compute types of the gather: T itself (FP64, FP32) or, for FP64 inputs in
// the mixed form, dfl: the weight products and the face sums carried as
// double-float pairs (relative 2^-44) on the FP32 pipe, GB300's FP64 pipe
// being 1/64 of it. Inputs are split exactly by integer operations
// (df_split), the sum goes back to FP64 with one addition per face.
struct dfl {
    df2 v;
};
__device__ __forceinline__ dfl operator*(dfl a, dfl b) { return dfl{df_mul(a.v, b.v)}; }
__device__ __forceinline__ dfl& operator+=(dfl& a, dfl b) {
    a.v = df_add(a.v, b.v);
    return a;
}
template <typename TC>
__device__ __forceinline__ TC tc_from(double v) { return TC(v); }
template <>
__device__ __forceinline__ dfl tc_from<dfl>(double v) { return dfl{df_split(v)}; }
template <typename T, typename TC>
__device__ __forceinline__ T tc_to(TC v) { return T(v); }
template <>
__device__ __forceinline__ double tc_to<double, dfl>(dfl v) { return f32_to_f64(v.v.hi) + f32_to_f64(v.v.lo); }

// Running sum of double-float products: an exact two-sum of the leading words and
// a plain sum of the trailing ones. Over the spreading's parts (60 terms at most per
// half warp, then pair additions) its error is no larger than that of a chain of pair
// additions: rms of the terms' sum of magnitudes, weights and forces of random sign,
// 8 terms 1.4e-14 and 1.5e-14, 400 terms 2.9e-15 and 3.0e-15, 6000 7.8e-16 and 1.7e-15.
struct alignas(8) DfAcc {
    float s, e;  // leading sum (two-summed), trailing sum
};
__device__ __forceinline__ void dfacc_add(DfAcc& a, float p, float pe) {
    const float s = a.s + p;
    const float v = s - a.s;
    a.e += ((a.s - (s - v)) + (p - v)) + pe;
    a.s = s;
}
__device__ __forceinline__ void dfacc_mul_add(DfAcc& a, df2 x, df2 y) {
    const float p = x.hi * y.hi;
    float e = fmaf(x.hi, y.hi, -p);
    e = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, e));
    dfacc_add(a, p, e);
}
__device__ __forceinline__ df2 dfacc_pair(DfAcc a) {
    df2 r;
    r.hi = a.s + a.e;
    r.lo = a.e - (r.hi - a.s);
    return r;
}

// ---------------------------------------------------------------------------
// Spreading. One block per active output tile of TS x TS x TZ faces and
// component (taken from a counter: their costs differ widely near a membrane).
// The markers binned in E = the tile grown by two cells per side are staged in
// shared memory in E-cell order (x fastest): every E row (ey, ez) is at most
// three contiguous runs of the sorted markers, one per x tile, and one block
// scan of the run lengths places them. The face planes of the tile each walk
// the staged markers whose cells lie within reach, a contiguous range; the
// ranges of all planes laid end to end are cut into equal shares for the warps.
// A warp walks its part of a plane with a half warp per marker and a lane per
// face of the marker's 4 x 4 footprint in the plane, into sums in shared
// memory (one copy per half warp), and leaves them in the slot of (plane,
// warp); after a barrier each plane's slots are added in warp order. No float
// atomics and a fixed order: bitwise repeatable. More markers than `cap` are
// taken in chunks of cap, the later ones added to the tile's faces in global
// memory: there is no marker-density limit.
//
// Bound by issue and shared-memory latency of the walks (FP64: by the FP64
// pipe as well, one instruction per marker, plane and half of the staged
// products). The form before gave each face a thread that searched the runs
// within its reach: 25 rows per face and component, a few markers each, most of
// them out of its support, so its lanes diverged. One warp per plane without
// the equal shares waited at the barrier for half its time (ncu). Measured at
// 256^3, 200,000 markers on shells: FP64 1397 -> 448 us, double-float
// 980 -> 497 us.
// ---------------------------------------------------------------------------
constexpr int kSpreadWarps = 8;
constexpr int kSpreadCap = 192;  // FP64 or double-float markers staged at once
// Resident blocks per SM that the registers are capped for and the grid counts on; 8^3
// tiles of FP64 or double-float values take 47 KB of shared memory, which leaves four.
constexpr int kSpreadBlocks = 5;
// values staged per marker: 4 x weights, and the products of 4 z and 4 y weights
// with the force
constexpr int kSpreadVals = 4 + 16;

// face sums of the compute type TC: acc += a b, and the value of two of them
template <typename TC>
struct FaceSum {
    typedef TC type;
    static __device__ __forceinline__ type zero() { return TC(0); }
    static __device__ __forceinline__ void madd(type& s, TC a, TC b) { s += a * b; }
    static __device__ __forceinline__ TC total(type a, type b) { return a + b; }
    static __device__ __forceinline__ TC add(TC a, TC b) { return a + b; }
};
template <>
struct FaceSum<dfl> {
    typedef DfAcc type;
    static __device__ __forceinline__ type zero() { return DfAcc{0.f, 0.f}; }
    static __device__ __forceinline__ void madd(type& s, dfl a, dfl b) { dfacc_mul_add(s, a.v, b.v); }
    static __device__ __forceinline__ dfl total(type a, type b) { return dfl{df_add(dfacc_pair(a), dfacc_pair(b))}; }
    static __device__ __forceinline__ dfl add(dfl a, dfl b) { return dfl{df_add(a.v, b.v)}; }
};

template <typename T, int TS, int TZ, typename TC = T>
__global__ void __launch_bounds__(32 * kSpreadWarps, kSpreadBlocks)
    k_spread_tiles(Dims d, int M, const int* __restrict__ perm, MarkerW<T> mw, const T* __restrict__ G,
                   const double* __restrict__ vol, double scale, const int* __restrict__ slot,
                   const int* __restrict__ ctab, const int* __restrict__ list, const int* __restrict__ count, int cap,
                   T* __restrict__ fu, T* __restrict__ fv, T* __restrict__ fw, int* __restrict__ next_item) {
    wait_launch();
    // 3D: TZ == TS, the neighbourhood grows by 2 cells per side along every
    // axis. 2D (TZ == 1, nz == 1): one plane, no z halo.
    constexpr int NW = kSpreadWarps, NT = 32 * NW, E = TS + 4, EZ = TZ == 1 ? 1 : TS + 4, HZ = TZ == 1 ? 0 : 2;
    constexpr int C = TS * TS * TZ, PL = TS * TS, SLOTS = NW + TZ - 1;
    constexpr int NSEG = 3 * E * EZ, SPT = (NSEG + NT - 1) / NT;  // runs, consecutive runs per thread
    typedef FaceSum<TC> FS;
    typedef typename FS::type Sum;
    extern __shared__ __align__(16) unsigned char smem[];
    TC* const s_w = (TC*)smem;                                   // [cap][kSpreadVals]
    Sum* const s_acc = (Sum*)(s_w + (size_t)cap * kSpreadVals);  // [warps][2][PL]
    TC* const s_part = (TC*)(s_acc + NW * 2 * PL);               // [SLOTS][PL]: sums of (plane, warp) at plane + warp
    int* const s_k = (int*)(s_part + SLOTS * PL);                // [cap]: marker of each staged slot
    unsigned* const s_b = (unsigned*)(s_k + cap);                // [cap]: packed footprint of each staged marker
    __shared__ int s_warp[NW], s_z[EZ + 1], s_li;
    const int ntx = d.nx / TS, nty = d.ny / TS;
    const int nitem = 3 * *count;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto wrap1 = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
    for (;;) {
        __syncthreads();
        if (tid == 0) s_li = atomicAdd(next_item, 1);
        __syncthreads();
        const int li = s_li;
        if (li >= nitem) break;
        const int t = list[li / 3], comp = li % 3;
        const int tx = t % ntx, ty = (t / ntx) % nty, tz = t / (ntx * nty);
        const int ox = tx * TS - 2, oy = ty * TS - 2, oz = tz * TZ - HZ;  // E origin (unwrapped cells)
        // ---- this thread's runs: sorted positions [p0, p0 + cnt)
        int p0[SPT], cnt[SPT], tot = 0;
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            const int sg = tid * SPT + k;
            p0[k] = cnt[k] = 0;
            if (sg < NSEG) {
                const int part = sg % 3, row = sg / 3, ey = row % E, ez = row / E;
                const int gy = oy + ey;
                if (!(d.channel && (gy < 0 || gy >= d.ny))) {
                    const int gyw = wrap1(gy, d.ny), gz = wrap1(oz + ez, d.nz);
                    const int txs = wrap1(tx + part - 1, ntx);
                    const int sl = slot[txs + ntx * (gyw / TS + nty * (gz / TZ))];
                    if (sl >= 0) {
                        const int x0 = part == 0 ? TS - 2 : 0, len = part == 1 ? TS : 2;
                        const int* r = ctab + (size_t)sl * (C + 1) + x0 + TS * ((gyw % TS) + TS * (gz % TZ));
                        p0[k] = r[0];
                        cnt[k] = r[len] - p0[k];
                    }
                }
            }
            tot += cnt[k];
        }
        // ---- block exclusive scan of the totals (thread order = E order)
        int inc = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        int off = inc - tot, nall = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if (w < warp) off += s_warp[w];
            nall += s_warp[w];
        }
        // an active tile whose neighbourhood holds no marker (its occupied
        // neighbour tiles' markers lie beyond the 2-cell halo) adds nothing:
        // its faces keep the zeros the callers wrote (block-uniform)
        if (nall == 0) continue;
        {
            int o = off;
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                const int sg = tid * SPT + k;
                if (sg < NSEG && sg % (3 * E) == 0) s_z[sg / (3 * E)] = o;  // first staged marker of E plane ez
                o += cnt[k];
            }
            if (tid == 0) s_z[EZ] = nall;
        }
        const int vx = comp == 0 ? 0 : 1, vy = comp == 1 ? 0 : 1, vz = comp == 2 ? 0 : 1;  // face offsets
        for (int lo = 0; lo < nall; lo += cap) {
            const int nc = nall - lo < cap ? nall - lo : cap;
            __syncthreads();  // s_z is written; the previous chunk is done with the staged markers
            {
                int o = off - lo;  // this thread's first run, relative to the chunk
#pragma unroll
                for (int k = 0; k < SPT; ++k) {
                    const int m0 = o < 0 ? -o : 0, m1 = cnt[k] < nc - o ? cnt[k] : nc - o;
                    for (int m = m0; m < m1; ++m) s_k[o + m] = perm[p0[k] + m];
                    o += cnt[k];
                }
            }
            __syncthreads();
            // ---- the chunk's products, a marker's values on consecutive threads
            for (int i = tid; i < nc * 4; i += NT) {
                const int m = i >> 2, j = i & 3, k = s_k[m];
                const T* w = mw.w + (size_t)k * 24;
                TC* o = s_w + (size_t)m * kSpreadVals;
                double g = (double)G[(size_t)comp * M + k];
                if (vol) g *= vol[k];
                const TC wz = tc_from<TC>(w[16 + 4 * vz + j]) * tc_from<TC>(g);
                o[j] = tc_from<TC>(w[4 * vx + j]);
#pragma unroll
                for (int y = 0; y < 4; ++y) o[4 + 4 * j + y] = tc_from<TC>(w[8 + 4 * vy + y]) * wz;
            }
            // ---- and footprints: the lanes (4 iy + ix) whose faces lie in the tile, the face of lane 0
            //      within the plane (36 added) and the first face plane (8 added)
            for (int m = tid; m < nc; m += NT) {
                const int k = s_k[m];
                int f[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int o = a == 0 ? ox : (a == 1 ? oy : oz);
                    const int n_a = a == 0 ? d.nx : (a == 1 ? d.ny : d.nz);
                    int ec = mw.cell[3 * k + a] - o;  // E-local cell
                    if (!(a == 1 && d.channel)) ec = wrapi(ec, n_a);
                    f[a] = ec + mw.dbase[(k * 3 + a) * 2 + (a == comp ? 0 : 1)];  // E-local first face
                }
                unsigned mx = 0, mask = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) mx |= (unsigned)(f[0] + i - 2) < (unsigned)TS ? 1u << i : 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i) mask |= (unsigned)(f[1] + i - 2) < (unsigned)TS ? mx << (4 * i) : 0u;
                s_b[m] = mask | (unsigned)(f[0] - 2 + TS * (f[1] - 2) + 36) << 16 | (unsigned)(f[2] + 8) << 24;
            }
            __syncthreads();
            // ---- walks: E planes of cells within reach of face plane J = lz + HZ are [J - 2, J + 2]
            //      ([J - 2, J + 1] where the faces sit on integer z), the only one in 2D
            auto range = [&](int lz, int& m0, int& m1) {
                const int J = lz + HZ, e0 = TZ == 1 ? 0 : J - 2, e1 = TZ == 1 ? 0 : (comp == 2 ? J + 1 : J + 2);
                m0 = s_z[e0] - lo;
                m1 = s_z[e1 + 1] - lo;
                m0 = m0 > 0 ? m0 : 0;
                m1 = m1 < nc ? m1 : nc;
                if (m1 < m0) m1 = m0;
            };
            int visits = 0;
#pragma unroll
            for (int lz = 0; lz < TZ; ++lz) {
                int m0, m1;
                range(lz, m0, m1);
                visits += m1 - m0;
            }
            // warp w takes visits [share(w), share(w + 1)), even shares so that both halves work
            const int per = ((visits + 2 * NW - 1) / (2 * NW)) * 2;
            auto part_of = [&](int w, int first, int m0, int m1, int& a, int& b) {
                a = w * per - first;
                b = a + per;
                a = m0 + (a > 0 ? a : 0);
                b = m0 + (b < m1 - m0 ? b : m1 - m0);
                return a < b;
            };
            {
                Sum* const acc = s_acc + warp * 2 * PL;
                const int half = lane >> 4, l16 = lane & 15;
                Sum* const mine = acc + half * PL + (l16 & 3) + TS * (l16 >> 2) - 36;
                const TC* const wx0 = s_w + (l16 & 3);
                const TC* const wyz0 = s_w + 4 + (l16 >> 2);
                int first = 0;
                for (int lz = 0; lz < TZ; ++lz) {
                    int m0, m1, a, b;
                    range(lz, m0, m1);
                    if (part_of(warp, first, m0, m1, a, b)) {
                        for (int i = lane; i < 2 * PL; i += 32) acc[i] = FS::zero();
                        __syncwarp();
                        // this lane's term of marker m: its face sum, or null outside the plane or the tile
                        auto term = [&](int m, TC& x, TC& yz) -> Sum* {
                            if (m >= b) return nullptr;
                            const unsigned pk = s_b[m];
                            const unsigned kz = (unsigned)(lz + HZ + 8) - (pk >> 24);
                            if (kz >= 4u || !((pk >> l16) & 1u)) return nullptr;
                            x = wx0[m * kSpreadVals];
                            yz = wyz0[m * kSpreadVals + 4 * kz];
                            return mine + ((pk >> 16) & 255u);
                        };
                        // two markers of the half warp in flight: the second's loads do
                        // not wait for the first's sum
                        for (int m = a + half; m - half < b; m += 4) {
                            TC x0, y0, x1, y1;
                            Sum* const f0 = term(m, x0, y0);
                            Sum* const f1 = term(m + 2, x1, y1);
                            if (f0) FS::madd(*f0, x0, y0);
                            __syncwarp();
                            if (f1) FS::madd(*f1, x1, y1);
                            __syncwarp();
                        }
                        for (int i = lane; i < PL; i += 32) s_part[(lz + warp) * PL + i] = FS::total(acc[i], acc[PL + i]);
                        __syncwarp();
                    }
                    first += m1 - m0;
                }
            }
            __syncthreads();
            // ---- a plane's parts in warp order
            T* const out = comp == 0 ? fu : (comp == 1 ? fv : fw);
            int first = 0;
            for (int lz = 0; lz < TZ; ++lz) {
                int m0, m1;
                range(lz, m0, m1);
                if (lz % NW == warp)
                    for (int i = lane; i < PL; i += 32) {
                        TC v = tc_from<TC>(0.0);
                        for (int w = 0; w < NW; ++w) {
                            int a, b;
                            if (part_of(w, first, m0, m1, a, b)) v = FS::add(v, s_part[(lz + w) * PL + i]);
                        }
                        const int gx = tx * TS + i % TS, gy = ty * TS + i / TS, gz = tz * TZ + lz;
                        if (d.channel && comp == 1 && gy == 0) continue;  // the wall plane
                        const T r = T((double)tc_to<T, TC>(v) * scale);
                        T* const o = out + lin(d, gx, gy, gz);
                        *o = lo == 0 ? r : *o + r;
                    }
                first += m1 - m0;
            }
        }
    }
}

// Interpolation U_k = sum over 4^3 faces of (phi/n)^3 * u(face)
// (src/ib/grid.h:68-84 with volume h^3, src/ib/eulerian_grid.h:45).
template <typename T, typename TF>
__global__ void k_interp(Dims d, int M, const int* __restrict__ perm, MarkerW<T> mw, const TF* __restrict__ u,
                         const TF* __restrict__ v, const TF* __restrict__ w, double* __restrict__ U) {
    wait_launch();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const int k = perm ? perm[p] : p;
    const int ext[3] = {d.nx, d.ny, d.nz};
    for (int comp = 0; comp < 3; ++comp) {
        const TF* src = comp == 0 ? u : (comp == 1 ? v : w);
        int idx[3][4];
        T wt[3][4];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int var = (a == comp) ? 0 : 1;
            const int b = mw.cell[3 * k + a] + mw.dbase[(k * 3 + a) * 2 + var];
            const T* ww = mw.w + (((size_t)k * 3 + a) * 2 + var) * 4;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                idx[a][m] = wrapi(b + m, ext[a]);
                wt[a][m] = ww[m];
            }
        }
        T acc = T(0);
#pragma unroll
        for (int mz = 0; mz < 4; ++mz)
#pragma unroll
            for (int my = 0; my < 4; ++my) {
                const T wyz = wt[1][my] * wt[2][mz];
                const long long row = (long long)d.nx * (idx[1][my] + (long long)d.ny * idx[2][mz]);
#pragma unroll
                for (int mx = 0; mx < 4; ++mx) acc += wt[0][mx] * wyz * T(src[row + idx[0][mx]]);
            }
        U[(size_t)comp * M + k] = (double)acc;
    }
}

// The same interpolation of FP64 fields in double-float on the FP32 pipe
// (the mixed form; GB300's FP64 pipe runs at 1/64 of the FP32 rate). Four
// lanes take one marker, one x tap each: a lane issues the loads of its 16
// (y, z) faces of a component back to back (the fields are larger than L2,
// so the time is DRAM latency), sums them as sum_z wz sum_y wy u, takes its
// x weight, and the quad adds its four partial sums by shuffles in a fixed
// pattern (the first lane's result is stored). Field values and weights are
// split exactly by integer operations (df_split, 24 + 23 bits); each product
// is a pair (fma two-product plus the cross terms) and the sums keep an
// exact two-sum of the leading words and a plain sum of the trailing ones, so
// the result is within a few units of 2^-46 of the largest term times the 4
// to 16 terms of a sum. One FP64 addition per component turns the pair back
// into FP64.
constexpr int kInterpDfBlock = 128;

template <bool PAIRS>
__global__ void __launch_bounds__(kInterpDfBlock) k_interp_dfl(Dims d, int M, const int* __restrict__ perm,
                                                               MarkerW<double> mw, const double* __restrict__ u,
                                                               const double* __restrict__ v,
                                                               const double* __restrict__ w, const float* __restrict__ uh,
                                                               const float* __restrict__ ul,
                                                               const float* __restrict__ vh,
                                                               const float* __restrict__ vl,
                                                               const float* __restrict__ wh,
                                                               const float* __restrict__ wl, double* __restrict__ U) {
    wait_launch();
    const int p = (blockIdx.x * kInterpDfBlock + threadIdx.x) >> 2;
    const int q = threadIdx.x & 3;
    if (p >= M) return;  // a quad leaves together
    const unsigned qmask = 0xfu << (threadIdx.x & 28);
    const int k = perm ? perm[p] : p;
#pragma unroll 1
    for (int comp = 0; comp < 3; ++comp) {
        const double* src = comp == 0 ? u : (comp == 1 ? v : w);
        const int vx = comp == 0 ? 0 : 1, vy = comp == 1 ? 0 : 1, vz = comp == 2 ? 0 : 1;
        const int bx = mw.cell[3 * k] + mw.dbase[(k * 3 + 0) * 2 + vx];
        const int by = mw.cell[3 * k + 1] + mw.dbase[(k * 3 + 1) * 2 + vy];
        const int bz = mw.cell[3 * k + 2] + mw.dbase[(k * 3 + 2) * 2 + vz];
        const long long ix = wrapi(bx + q, d.nx);
        long long roff[4][4];
#pragma unroll
        for (int mz = 0; mz < 4; ++mz)
#pragma unroll
            for (int my = 0; my < 4; ++my)
                roff[mz][my] = (long long)d.nx * (wrapi(by + my, d.ny) + (long long)d.ny * wrapi(bz + mz, d.nz)) + ix;
        df2 val[4][4];
        if (PAIRS) {  // the velocity's float pairs (hi + lo), no splits
            const float* sh = comp == 0 ? uh : (comp == 1 ? vh : wh);
            const float* sl = comp == 0 ? ul : (comp == 1 ? vl : wl);
#pragma unroll
            for (int mz = 0; mz < 4; ++mz)
#pragma unroll
                for (int my = 0; my < 4; ++my) {
                    val[mz][my].hi = sh[roff[mz][my]];
                    val[mz][my].lo = sl[roff[mz][my]];
                }
        } else {
            double dv[4][4];
#pragma unroll
            for (int mz = 0; mz < 4; ++mz)
#pragma unroll
                for (int my = 0; my < 4; ++my) dv[mz][my] = src[roff[mz][my]];
#pragma unroll
            for (int mz = 0; mz < 4; ++mz)
#pragma unroll
                for (int my = 0; my < 4; ++my) val[mz][my] = df_split(dv[mz][my]);
        }
        // the quad's lanes split one y and one z weight each and share them
        const df2 wyq = df_split(mw.w[(((size_t)k * 3 + 1) * 2 + vy) * 4 + q]);
        const df2 wzq = df_split(mw.w[(((size_t)k * 3 + 2) * 2 + vz) * 4 + q]);
        const int q0 = threadIdx.x & 28;
        df2 wy[4], wz[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            wy[m].hi = __shfl_sync(qmask, wyq.hi, q0 + m);
            wy[m].lo = __shfl_sync(qmask, wyq.lo, q0 + m);
            wz[m].hi = __shfl_sync(qmask, wzq.hi, q0 + m);
            wz[m].lo = __shfl_sync(qmask, wzq.lo, q0 + m);
        }
        DfAcc az = {0.f, 0.f};
#pragma unroll
        for (int mz = 0; mz < 4; ++mz) {
            DfAcc ay = {0.f, 0.f};
#pragma unroll
            for (int my = 0; my < 4; ++my) dfacc_mul_add(ay, wy[my], val[mz][my]);
            dfacc_mul_add(az, wz[mz], dfacc_pair(ay));
        }
        const df2 wxq = df_split(mw.w[(((size_t)k * 3 + 0) * 2 + vx) * 4 + q]);
        df2 r = df_mul(wxq, dfacc_pair(az));
        df2 o;
        o.hi = __shfl_xor_sync(qmask, r.hi, 1);
        o.lo = __shfl_xor_sync(qmask, r.lo, 1);
        r = df_add(r, o);
        o.hi = __shfl_xor_sync(qmask, r.hi, 2);
        o.lo = __shfl_xor_sync(qmask, r.lo, 2);
        r = df_add(r, o);
        if (q == 0) U[(size_t)comp * M + k] = f32_to_f64(r.hi) + f32_to_f64(r.lo);
    }
}

// X_out = X_in + c * U  (U component-major)
__global__ void k_marker_axpy(int M, double* __restrict__ Xo, const double* __restrict__ Xi, const double* __restrict__ U,
                              double c) {
    wait_launch();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
#pragma unroll
    for (int a = 0; a < 3; ++a) Xo[3 * k + a] = Xi[3 * k + a] + c * U[(size_t)a * M + k];
}

}  // namespace

template <typename T>
void launch_springs_bending(int M, const double* X, const int* nstart, const int* nidx, double ks, double kb,
                            double* Y, T* G, cudaStream_t s) {
    if (M <= 0) return;
    launch_dep((M + 255) / 256, 256, 0, s, k_lap_aos, M, X, nstart, nidx, Y);
    launch_dep((M + 255) / 256, 256, 0, s, k_spring_bend<T>, M, Y, nstart, nidx, ks, kb, G);
}
template <typename T>
void launch_springs(int M, const double* X, const int* nstart, const int* nidx, double k, T* G, cudaStream_t s) {
    if (M > 0) launch_dep((M + 255) / 256, 256, 0, s, k_springs<T>, M, X, nstart, nidx, k, G);
}

template <typename T>
void launch_marker_prep(const Dims& d, int TS, int M, const double* X, unsigned* keys, int* vals, MarkerW<T> mw,
                        int* flag, cudaStream_t s, bool df_weights) {
    if (M <= 0) return;
    if (df_weights && sizeof(T) == sizeof(double))
        launch_dep((M + 255) / 256, 256, 0, s, k_marker_prep<T, true>, d, TS, M, X, keys, vals, mw, flag);
    else
        launch_dep((M + 255) / 256, 256, 0, s, k_marker_prep<T, false>, d, TS, M, X, keys, vals, mw, flag);
}

size_t radix_sort_temp_bytes(int n) {
    const int nblk = (n + RS_TILE - 1) / RS_TILE;
    return (size_t)256 * ((nblk > 0 ? nblk : 1) + 1) * sizeof(unsigned);  // and the digits' totals
}

void radix_sort_pairs(unsigned* keys, int* vals, unsigned* keys_alt, int* vals_alt, int n, int bits, unsigned* hist,
                      unsigned** keys_out, int** vals_out, cudaStream_t s) {
    const int nblk = (n + RS_TILE - 1) / RS_TILE;
    unsigned* ka = keys;
    unsigned* kb = keys_alt;
    int* va = vals;
    int* vb = vals_alt;
    for (int shift = 0; shift < bits && n > 0; shift += 8) {
        launch_dep(nblk, RS_THREADS, 0, s, k_rs_hist, ka, n, shift, hist, nblk);
        launch_dep(256 / (RS_THREADS / 32), RS_THREADS, 0, s, k_rs_scan, hist, nblk);
        launch_dep(nblk, RS_THREADS, 0, s, k_rs_scatter, ka, va, kb, vb, n, shift, hist, nblk);
        unsigned* tk = ka; ka = kb; kb = tk;
        int* tv = va; va = vb; vb = tv;
    }
    *keys_out = ka;
    *vals_out = va;
}

// One block up to RS_SMALL markers and 65536 tiles (it clears the tile ranges too): with
// the ranges 11.7, 16.7, 26.9 and 36.9 us for 512, 2048, 5120 and 8192 markers on 4096
// tiles against 32, 41, 42 and 42 in passes over all SMs with the memsets; 14.8, 20.5,
// 34.8 and 44.3 against 34, 44, 46 and 46 on 32768. At 9000 markers the passes win (45.2
// against 43.0, 53.4 against 46.8), and the line in tiles is where 8192 markers take as
// long (65536: 51.9 against 52.4; 131072: 61.7 against 52.6; on 262144 2048 do).
bool sort_bins_small_ok(int n, int ntiles) { return n > 0 && n <= RS_SMALL && ntiles <= 65536; }
void sort_bins_small(unsigned* keys, int* vals, int n, int bits, int cells_per_tile, int ntiles, int* tstart, int* tend,
                     int* counts, cudaStream_t s) {
    auto launch = [&](auto* kernel, int items) {
        const size_t smem = sizeof(unsigned) * ((size_t)RSS_THREADS * items + 256 * RSS_COLS + 32) +
                            sizeof(unsigned short) * (size_t)RSS_THREADS * items;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_dep(1, RSS_THREADS, smem, s, kernel, keys, vals, n, bits, cells_per_tile, ntiles, tstart, tend, counts);
    };
    if (n <= 2 * RSS_THREADS) launch(k_sort_small<2>, 2);
    else launch(k_sort_small<RSS_ITEMS>, RSS_ITEMS);
}

void launch_tile_ranges(const unsigned* keys, int M, int cells_per_tile, int* tstart, int* tend, cudaStream_t s) {
    if (M > 0) launch_dep((M + 255) / 256, 256, 0, s, k_tile_ranges, keys, M, cells_per_tile, tstart, tend);
}

void launch_tiles(int TS, int TZ, int ntx, int nty, int ntz, int channel, const unsigned* keys, const int* tstart,
                  const int* tend, int* list, int* count, int* slot, int* ctab, cudaStream_t s) {
    const int nt = ntx * nty * ntz, blocks = std::max(1, std::min((nt + kTileWarps - 1) / kTileWarps, 152 * 16));
    auto launch = [&](auto* kernel) {
        launch_dep(blocks, 32 * kTileWarps, 0, s, kernel, ntx, nty, ntz, channel, keys, tstart, tend, list, count,
                   slot, ctab);
    };
    if (TS == 8 && TZ == 8) launch(k_tiles<8, 8>);
    else if (TS == 4 && TZ == 4) launch(k_tiles<4, 4>);
    else if (TS == 8) launch(k_tiles<8, 1>);
    else launch(k_tiles<4, 1>);
}

template <typename T, int TS, int TZ, typename TC>
static void spread_launch(const Dims& d, int M, const int* perm, MarkerW<T> mw, const T* G, const double* vol,
                          double scale, const int* slot, const int* ctab, const int* list, const int* count,
                          int max_tiles, T* fu, T* fv, T* fw, int* next_tile, cudaStream_t s) {
    const int cap = kSpreadCap * 8 / (int)sizeof(TC);
    const size_t smem = sizeof(TC) * ((size_t)cap * kSpreadVals + (3 * kSpreadWarps + TZ - 1) * TS * TS) + 8 * (size_t)cap;
    cudaFuncSetAttribute(k_spread_tiles<T, TS, TZ, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int blocks = std::max(1, std::min(3 * max_tiles, 152 * kSpreadBlocks));
    launch_dep(blocks, 32 * kSpreadWarps, smem, s, k_spread_tiles<T, TS, TZ, TC>, d, M, perm, mw, G, vol, scale,
               slot, ctab, list, count, cap, fu, fv, fw, next_tile);
}

template <typename T>
void launch_spread(const Dims& d, int TS, int M, const int* perm, MarkerW<T> mw, const T* G, const double* vol,
                   double scale, const int* slot, const int* ctab, const int* list, const int* count, int max_tiles,
                   T* fu, T* fv, T* fw, int* next_tile, cudaStream_t s, bool dfloat) {
    const bool flat = d.nz == 1;
#define AFMIB_SPREAD(TSV, TZV)                                                                                     \
    do {                                                                                                           \
        if (dfloat && sizeof(T) == sizeof(double))                                                                 \
            spread_launch<T, TSV, TZV, std::conditional_t<sizeof(T) == sizeof(double), dfl, T>>(                   \
                d, M, perm, mw, G, vol, scale, slot, ctab, list, count, max_tiles, fu, fv, fw, next_tile, s);      \
        else                                                                                                       \
            spread_launch<T, TSV, TZV, T>(d, M, perm, mw, G, vol, scale, slot, ctab, list, count, max_tiles, fu,   \
                                          fv, fw, next_tile, s);                                                   \
    } while (0)
    if (TS == 8 && !flat) AFMIB_SPREAD(8, 8);
    else if (TS == 4 && !flat) AFMIB_SPREAD(4, 4);
    else if (TS == 8) AFMIB_SPREAD(8, 1);
    else AFMIB_SPREAD(4, 1);
#undef AFMIB_SPREAD
}

template <typename T, typename TF>
void launch_interp(const Dims& d, int M, const int* perm, MarkerW<T> mw, const TF* u, const TF* v, const TF* w, double* U,
                   cudaStream_t s) {
    if (M > 0) launch_dep((M + 127) / 128, 128, 0, s, k_interp<T, TF>, d, M, perm, mw, u, v, w, U);
}

void launch_interp_dfl(const Dims& d, int M, const int* perm, MarkerW<double> mw, const double* u, const double* v,
                       const double* w, double* U, cudaStream_t s, const float* uh, const float* ul, const float* vh,
                       const float* vl, const float* wh, const float* wl) {
    if (M <= 0) return;
    const int blocks = (int)((4LL * M + kInterpDfBlock - 1) / kInterpDfBlock);
    if (uh && ul && vh && vl && wh && wl)
        launch_dep(blocks, kInterpDfBlock, 0, s, k_interp_dfl<true>, d, M, perm, mw, u, v, w, uh, ul, vh, vl, wh, wl,
                   U);
    else
        launch_dep(blocks, kInterpDfBlock, 0, s, k_interp_dfl<false>, d, M, perm, mw, u, v, w, nullptr, nullptr,
                   nullptr, nullptr, nullptr, nullptr, U);
}

void launch_marker_axpy(int M, double* Xo, const double* Xi, const double* U, double c, cudaStream_t s) {
    if (M > 0) launch_dep((M + 255) / 256, 256, 0, s, k_marker_axpy, M, Xo, Xi, U, c);
}

#define AFMIB_IB_INST(T)                                                                                        \
    template void launch_springs<T>(int, const double*, const int*, const int*, double, T*, cudaStream_t);       \
    template void launch_springs_bending<T>(int, const double*, const int*, const int*, double, double, double*, T*, \
                                            cudaStream_t);                                                         \
    template void launch_marker_prep<T>(const Dims&, int, int, const double*, unsigned*, int*, MarkerW<T>, int*, \
                                        cudaStream_t, bool);                                                     \
    template void launch_spread<T>(const Dims&, int, int, const int*, MarkerW<T>, const T*, const double*, double,  \
                                   const int*, const int*, const int*, const int*, int, T*, T*, T*, int*,           \
                                   cudaStream_t, bool);                                                             \
    template void launch_interp<T, double>(const Dims&, int, const int*, MarkerW<T>, const double*, const double*, \
                                           const double*, double*, cudaStream_t);                               \
    template void launch_interp<T, float>(const Dims&, int, const int*, MarkerW<T>, const float*, const float*,  \
                                          const float*, double*, cudaStream_t);

AFMIB_IB_INST(double)
AFMIB_IB_INST(float)

}  // namespace afmib
