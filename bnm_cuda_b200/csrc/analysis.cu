// FC, sliding-window FC, FCD, KS distance and goodness of fit on the device.
//
// Reference behaviour (CPU path, which the GPU reference approximates):
//   FC          check_fit.cpp:19-62   Pearson over kept frames, pairs i>j in
//                                    row order, optional inter-hemispheric skip
//   window FC   check_fit.cpp:79-106  windows centred ws/2 .. n-1-ws/2 by step,
//                                    [c-ws/2, c+ws/2] inclusive
//   FCD         check_fit.cpp:110-134 Pearson between window-FC vectors, i>j
//   KS          check_fit.cpp:202-210 two-sample KS of emp vs sim FCD (libks)
//   GOF         check_fit.cpp:171-215 1 - r(FC) + |dmean FC| + KS; NaN -> MAX_COST
//   FIC penalty bnm.cpp:389-405, bnm.cu:752-767
//
// B200 layout:
//   * fc_window_kernel: one CTA per (tile of node pairs, simulation).  BOLD
//     frames stream through a shared-memory ring as centred FP64 values; every
//     pair keeps FP64 running co-moments, updated by one add and one subtract
//     per frame as the window slides, so window FC costs O(P) per window
//     instead of O(P*L).  Static FC comes from the same pass.  Window
//     sums over pairs (for the FCD centring) are formed from the finished rows
//     in FP64 in a fixed order, so the FCD does not depend on the window tile.
//   * fcd_gram_kernel: FCD = Z Z^T over the centred, unit-norm window-FC rows
//     (FP32), lower triangle only; its epilogue drops each
//     FCD value into the KS histogram (upper_bound rank among the sorted
//     empirical FCD), so FCD never has to be sorted.
//   * gof_kernel: prefix-scan of that histogram (a cluster of CTAs per
//     simulation) gives the exact KS statistic;
//     FC correlation / mean difference in FP64; cost assembly.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#include "cluster_util.cuh"
#include "kernels.h"

namespace bnm {


__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ------------------------------------------------------------ window FC
//
// Threads: 256 that own RI x RJ pairs each (thread (ty, tx): nodes i0 + ty +
// 16 a and j0 + tx + 16 b), and one per node of the tile (its 16 RI rows and
// 16 RJ columns) that centres the node's series, writes it to the ring and
// keeps the node's window sums, a chunk of kChunk frames ahead of the pairs.
//
// What bounds it: the FP64 pipe, about 15 operations a pair and window (three
// co-moment updates, the covariance, and the quotient below), at 16 lanes per
// cycle of an SM quarter.  The former kernel took pairs from a table: each
// read four series values and converted and centred them itself, every frame
// cost two block barriers, and the quotient was CUDA's square root and
// division, a branch each: 7.6 ms at N = 400, 4 series of 1201 frames (79,800
// pairs, 1157 windows; now 1.3 ms), 1.35 ms at N = 100, 64 series of 585
// frames (now 0.63 ms).
constexpr int kChunk = 8;

// (float)(cov / sqrt(vi vj)) as the plain FP64 expression gives it.
__device__ __noinline__ double corr_plain(double cov, double vi, double vj) { return cov / sqrt(vi * vj); }
// The same FP32 value without the branches of the division and square root:
// the product with a reciprocal root from two Newton steps is within 2^-50 of
// the plain expression, so both round to the same FP32 value unless that
// interval holds the midpoint of two FP32 neighbours, or the value is below
// FP32's normal range; those have to be done over (redo).  vi and vj inside
// var_ok's range.
__device__ __forceinline__ double corr_fast(double cov, double vi, double vj, bool& redo) {
    const double p = vi * vj, h = 0.5 * p;
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p));
    y = fma(y, fma(-h, y * y, 0.5), y);
    y = fma(y, fma(-h, y * y, 0.5), y);
    const double r = cov * y;
    const unsigned lo = ((unsigned)__double2loint(r) - (0x10000000u - 128u)) & 0x1fffffffu;  // bits below FP32's last
    redo = lo <= 256u || ((unsigned)__double2hiint(r) & 0x7fffffffu) < 0x38200000u;            // |r| < 2^-125
    return r;
}
// 2^-450 <= v < 2^450: products and their reciprocal roots keep full precision
__device__ __forceinline__ bool var_ok(double v) {
    return (unsigned)__double2hiint(v) - 0x23d00000u < 0x5c100000u - 0x23d00000u;
}

// Shared memory: ring [rl][NT] double, window sums [2][kChunk][NT] double2
// (sum, variance sum), node means [NT], series sums [NT] double2, and per
// window slot whether a variance was outside var_ok's range (int [2][kChunk + 1],
// the last for the series).
template <typename TB, int RI, int RJ, bool kRing>
__global__ void __launch_bounds__(256 + (RI + RJ + 1) / 2 * 32) fc_window_kernel(FcArgs a, const TB* __restrict__ bold,
                                                                                 int rl) {
    constexpr int TI = 16 * RI, TJ = 16 * RJ, NT = TI + TJ;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* ring = reinterpret_cast<double*>(smem_raw);
    double2* stat = reinterpret_cast<double2*>(ring + (size_t)rl * NT);
    double2* series = stat + 2 * kChunk * NT;
    double* mean = reinterpret_cast<double*>(series + NT);
    int* odd = reinterpret_cast<int*>(mean + NT);
    for (int e = threadIdx.x; e < 2 * (kChunk + 1); e += blockDim.x) odd[e] = 0;
    __syncthreads();

    // the tile: group (hemisphere with exc, else all nodes), row block, column
    // block; only tiles with pairs j < i exist
    const int M = a.exc ? a.N / 2 : a.N;
    int tile = blockIdx.y, g0 = 0, bi = 0;
    for (;; bi++) {
        if (bi * TI >= M) {
            g0 += M;
            bi = 0;
        }
        const int imax = min((bi + 1) * TI, M) - 1, nb = imax < 1 ? 0 : (imax - 1) / TJ + 1;
        if (tile < nb) break;
        tile -= nb;
    }
    const int i0 = g0 + bi * TI, j0 = g0 + tile * TJ, gend = g0 + M;
    const int N = a.N, L = a.win_len, T0 = a.corr_len, W = a.W, step = a.win_step, sim = blockIdx.x;
    const TB* src = bold + ((size_t)sim * a.frames + a.n_vols_remove) * N;
    const double invL = 1.0 / L, invT = 1.0 / T0;
    const int chunks = (T0 + kChunk - 1) / kChunk;
    int k = 0, lo = 0;  // current window and the first frame it covers

    if (threadIdx.x >= 256) {  // ---- one thread per node of the tile ----
        const int n = threadIdx.x - 256;
        const int node = n < TI ? i0 + n : j0 + n - TI;
        const bool on = n < NT && node < gend;
        const TB* x = src + (on ? node : i0);
        double s = 0.0;
        int t = 0;
        // FP64 sum in frame order; the pairs wait for it, so many loads at once
        // (eight: 0.4 us a round of them, 14 of 76 us of the kernel at 271
        // frames, 4 x 68 nodes; now 70 us; 300 x 30 nodes 134 -> 123 us; with
        // more waves of CTAs they hide it for one another)
        constexpr int kAtOnce = 128 / sizeof(TB);
        for (; t + kAtOnce <= T0; t += kAtOnce) {
            TB v[kAtOnce];
#pragma unroll
            for (int u = 0; u < kAtOnce; u++) v[u] = x[(size_t)(t + u) * N];
#pragma unroll
            for (int u = 0; u < kAtOnce; u++) s += (double)v[u];
        }
        if (t < T0) {
            TB v[kAtOnce];
#pragma unroll
            for (int u = 0; u < kAtOnce; u++) v[u] = x[(size_t)min(t + u, T0 - 1) * N];
#pragma unroll
            for (int u = 0; u < kAtOnce; u++)
                if (t + u < T0) s += (double)v[u];
        }
        const double mu = s / T0;
        if (n < NT) mean[n] = mu;
        double fs = 0.0, fss = 0.0, ws = 0.0, wss = 0.0;
        TB v[kChunk];
        auto fetch = [&](int c) {
#pragma unroll
            for (int f = 0; f < kChunk; f++) v[f] = x[(size_t)min(c * kChunk + f, T0 - 1) * N];
        };
        fetch(0);
        int pos = 0;  // ring slot of frame t
        for (int c = 0; c <= chunks; c++) {
            if (c < chunks && n < NT) {
                double y[kChunk];
#pragma unroll
                for (int f = 0; f < kChunk; f++) y[f] = (double)v[f] - mu;
                if (c + 1 < chunks) fetch(c + 1);
                int slot = 0;
#pragma unroll
                for (int f = 0; f < kChunk; f++) {
                    const int t = c * kChunk + f;
                    if (t >= T0) break;
                    ring[pos * NT + n] = y[f];
                    fs += y[f];
                    fss = fma(y[f], y[f], fss);
                    if (k < W && t >= lo) {
                        ws += y[f];
                        wss = fma(y[f], y[f], wss);
                    }
                    if (k < W && t == k * step + L - 1) {
                        const double v = fma(-(ws * ws), invL, wss);
                        stat[((c & 1) * kChunk + slot) * NT + n] = make_double2(ws, v);
                        // a window's flag is never cleared: from then on its slot takes the plain path
                        if (on && !var_ok(v)) odd[(c & 1) * kChunk + slot] = 1;
                        slot++;
                        // slide to window k + 1: drop the frames it no longer covers
                        const int nlo = (k + 1) * step;
                        if (nlo <= t) {
                            for (int tt = lo; tt < nlo; tt++) {
                                int q = pos - (t - tt);
                                if (q < 0) q += rl;
                                const double yl = kRing ? ring[q * NT + n] : (double)x[(size_t)tt * N] - mu;
                                ws -= yl;
                                wss = fma(-yl, yl, wss);
                            }
                        } else {
                            ws = wss = 0.0;
                        }
                        lo = nlo;
                        k++;
                    }
                    if (++pos == rl) pos = 0;
                }
                if (c == chunks - 1) {
                    const double v = fma(-(fs * fs), invT, fss);
                    series[n] = make_double2(fs, v);
                    if (on && !var_ok(v)) odd[2 * kChunk] = 1;
                }
            }
            __syncthreads();  // chunk c is ready, chunk c - 1 has been used
        }
        return;
    }

    // ---- pairs ----
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double full[RI][RJ], win[RI][RJ];
    bool pv[RI][RJ];
    int pidx[RI];  // pair index of (i, j) = pidx + j
#pragma unroll
    for (int u = 0; u < RI; u++) {
        const int i = i0 + ty + 16 * u, r = i - g0;  // rows before i in its group hold r (r - 1) / 2 pairs
        pidx[u] = (g0 ? M * (M - 1) / 2 : 0) + r * (r - 1) / 2 - g0;
#pragma unroll
        for (int w = 0; w < RJ; w++) {
            pv[u][w] = i < gend && j0 + tx + 16 * w < i;
            full[u][w] = win[u][w] = 0.0;
        }
    }
    bool any_nan = false;
    // correlations of the tile from co-moments m and node sums st, to `to`
    auto emit = [&](const double (&m)[RI][RJ], const double2* st, double inv, bool plain, float* to) {
        double2 si[RI], sj[RJ];
#pragma unroll
        for (int u = 0; u < RI; u++) si[u] = st[ty + 16 * u];
#pragma unroll
        for (int w = 0; w < RJ; w++) sj[w] = st[TI + tx + 16 * w];
        unsigned again = 0;
#pragma unroll
        for (int u = 0; u < RI; u++)
#pragma unroll
            for (int w = 0; w < RJ; w++) {
                bool redo;
                const double cov = fma(-(si[u].x * sj[w].x), inv, m[u][w]);
                const double r = corr_fast(cov, si[u].y, sj[w].y, redo);
                if (pv[u][w]) to[pidx[u] + 16 * w] = (float)r;
                again |= redo && pv[u][w] ? 1u << (u * RJ + w) : 0u;
            }
        if (!again && !plain) return;
#pragma unroll
        for (int u = 0; u < RI; u++)
#pragma unroll
            for (int w = 0; w < RJ; w++) {
                if (!pv[u][w] || !(plain || (again >> (u * RJ + w) & 1))) continue;
                const double cov = fma(-(si[u].x * sj[w].x), inv, m[u][w]);
                const double r = corr_plain(cov, si[u].y, sj[w].y);
                if (!(r == r) || isinf(r)) any_nan = true;
                to[pidx[u] + 16 * w] = (float)r;
            }
    };
    const double* yi = ring + ty;
    const double* yj = ring + TI + tx;
    float* out = a.wfc + (size_t)sim * W * a.P + j0 + tx;
    __syncthreads();  // chunk 0
    int pos = 0, lpos = 0;  // ring slots (as offsets) of frame t and of frame lo
    const int rend = rl * NT;
    int t_out = L - 1;  // last frame of window k
    for (int c = 0; c < chunks; c++) {
        int slot = (c & 1) * kChunk;
        const int t1 = min(T0, (c + 1) * kChunk);
        for (int t = c * kChunk; t < t1; t++) {
            const bool in_win = k < W && t >= lo;
            double ei[RI], ej[RJ];
#pragma unroll
            for (int u = 0; u < RI; u++) ei[u] = yi[pos + 16 * u];
#pragma unroll
            for (int w = 0; w < RJ; w++) ej[w] = yj[pos + 16 * w];
#pragma unroll
            for (int u = 0; u < RI; u++)
#pragma unroll
                for (int w = 0; w < RJ; w++) {
                    full[u][w] = fma(ei[u], ej[w], full[u][w]);
                    if (in_win) win[u][w] = fma(ei[u], ej[w], win[u][w]);
                }
            if (k < W && t == t_out) {
                emit(win, stat + slot * NT, invL, odd[slot] != 0, out);
                slot++;
                out += a.P;
                const int nlo = lo + step;
                if (nlo <= t) {
                    for (int tt = lo; tt < nlo; tt++) {
                        double li[RI], lj[RJ];
                        if (kRing) {
#pragma unroll
                            for (int u = 0; u < RI; u++) li[u] = yi[lpos + 16 * u];
#pragma unroll
                            for (int w = 0; w < RJ; w++) lj[w] = yj[lpos + 16 * w];
                            lpos += NT;
                            if (lpos == rend) lpos = 0;
                        } else {
                            const TB* x = src + (size_t)tt * N;
#pragma unroll
                            for (int u = 0; u < RI; u++)
                                li[u] = (double)x[min(i0 + ty + 16 * u, gend - 1)] - mean[ty + 16 * u];
#pragma unroll
                            for (int w = 0; w < RJ; w++)
                                lj[w] = (double)x[min(j0 + tx + 16 * w, gend - 1)] - mean[TI + tx + 16 * w];
                        }
#pragma unroll
                        for (int u = 0; u < RI; u++)
#pragma unroll
                            for (int w = 0; w < RJ; w++) win[u][w] = fma(-li[u], lj[w], win[u][w]);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < RI; u++)
#pragma unroll
                        for (int w = 0; w < RJ; w++) win[u][w] = 0.0;
                    if (kRing) lpos = nlo % rl * NT;
                }
                lo = nlo;
                t_out += step;
                k++;
            }
            pos += NT;
            if (pos == rend) pos = 0;
        }
        __syncthreads();  // this chunk's ring slots and sums may be refilled
    }
    // static FC over all kept frames
    emit(full, series, invT, odd[2 * kChunk] != 0, a.fc + (size_t)sim * a.P + j0 + tx);
    if (any_nan) atomicOr(&a.nan_flag[sim], 1);
}

// ---------------------------------------------------------------- FCD Gram

// kTile x kTile outputs per CTA, RT x RT per thread (16 x 16 threads).  K
// chunks are normalised (FP64) into one of two shared buffers while the other
// is used; their loads are in flight two chunks ahead.  Every output's sum runs
// over K in order, so K cannot be split.  What bounds it: with few tiles the
// chain of a chunk (load, conversion, barrier) on an SM with one CTA, with many
// the shared-memory reads, which are four K at a time (rows of 36 floats: the
// 16-byte reads of 8 rows touch all banks once).  Few simulations with few
// windows leave most SMs without a 64 x 64 tile, so those take 32 x 32.
// Measured with the window sums, one K per read -> now: 4 x 121 windows of
// 1122 pairs (32 x 32) 56 -> 42 us, 2 x 136 of 39,800 1.48 -> 0.98 ms; 64 x 278
// of 2450 (64 x 64) 1.20 -> 0.92 ms.
constexpr int kTk = 32;

template <int kTile>
__global__ void __launch_bounds__(256, 2) fcd_gram_kernel(FcdArgs a) {
    constexpr int RT = kTile / 16, kLoads = kTile * kTk / 256;
    // blockIdx.x: lower-triangular tile index, blockIdx.y: simulation
    int t = blockIdx.x, ta = 0;
    while (t >= ta + 1) { t -= ta + 1; ta++; }
    const int tb = t;  // ta >= tb
    const int sim = blockIdx.y;
    __shared__ __align__(16) float As[2][kTile][kTk + 4];
    __shared__ __align__(16) float Bs[2][kTile][kTk + 4];
    __shared__ double mA[kTile], sA[kTile], mB[kTile], sB[kTile];
    const int a0 = ta * kTile, b0 = tb * kTile;
    const float* V = a.wfc + (size_t)sim * a.W * a.P;
    const double* ws = a.wsum + (size_t)sim * a.W * 2;
    if (threadIdx.x < kTile) {
        const int r = a0 + threadIdx.x;
        double m = 0, s = 0;
        if (r < a.W) window_norm(ws + 2 * r, a.p1 - a.p0, m, s);
        mA[threadIdx.x] = m;
        sA[threadIdx.x] = s;
    } else if (threadIdx.x < 2 * kTile) {
        const int r = b0 + threadIdx.x - kTile;
        double m = 0, s = 0;
        if (r < a.W) window_norm(ws + 2 * r, a.p1 - a.p0, m, s);
        mB[threadIdx.x - kTile] = m;
        sB[threadIdx.x - kTile] = s;
    }
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int lc = threadIdx.x % kTk, lr = threadIdx.x / kTk;  // column of this thread's loads, first row
    constexpr int kStep = 256 / kTk;
    float v[2][2][kLoads];  // [chunk parity][A, B]
    // no branch around a load or a conversion: the addresses are clamped, the
    // values outside the rows and the pair range are replaced by zeros
    auto fetch = [&](float (&v)[2][kLoads], int k0) {
        const float* p = V + min(k0 + lc, a.p1 - 1);
#pragma unroll
        for (int e = 0; e < kLoads; e++) {
            v[0][e] = p[(size_t)min(a0 + lr + e * kStep, a.W - 1) * a.P];
            v[1][e] = p[(size_t)min(b0 + lr + e * kStep, a.W - 1) * a.P];
        }
    };
    auto store = [&](const float (&v)[2][kLoads], int buf, int k0) {  // centred and scaled
        const bool in = k0 + lc < a.p1;
#pragma unroll
        for (int e = 0; e < kLoads; e++) {
            const int r = lr + e * kStep;
            const float x = (float)(((double)v[0][e] - mA[r]) * sA[r]), y = (float)(((double)v[1][e] - mB[r]) * sB[r]);
            As[buf][r][lc] = in && a0 + r < a.W ? x : 0.f;
            Bs[buf][r][lc] = in && b0 + r < a.W ? y : 0.f;
        }
    };
    float acc[RT][RT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < RT; j++) acc[i][j] = 0.f;
    auto multiply = [&](int buf) {
#pragma unroll 2
        for (int c = 0; c < kTk; c += 4) {
            float4 av[RT], bv[RT];
#pragma unroll
            for (int i = 0; i < RT; i++) av[i] = *reinterpret_cast<const float4*>(&As[buf][ty * RT + i][c]);
#pragma unroll
            for (int j = 0; j < RT; j++) bv[j] = *reinterpret_cast<const float4*>(&Bs[buf][tx + 16 * j][c]);
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < RT; j++) {
                    acc[i][j] = fmaf(av[i].x, bv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(av[i].y, bv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(av[i].z, bv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(av[i].w, bv[j].w, acc[i][j]);
                }
        }
    };
    fetch(v[0], a.p0);
    fetch(v[1], a.p0 + kTk);
    store(v[0], 0, a.p0);
    __syncthreads();
    for (int k0 = a.p0;;) {  // chunk k0 is in buffer 0, the next in v[1]
        fetch(v[0], k0 + 2 * kTk);
        multiply(0);
        if ((k0 += kTk) >= a.p1) break;
        store(v[1], 1, k0);
        __syncthreads();
        fetch(v[1], k0 + 2 * kTk);
        multiply(1);
        if ((k0 += kTk) >= a.p1) break;
        store(v[0], 0, k0);
        __syncthreads();
    }
    bool any_nan = false;
    unsigned int* hist = a.hist ? a.hist + (size_t)sim * (a.m + 1) : nullptr;
    unsigned int* eq = a.hist ? a.eq + (size_t)sim * (a.m + 1) : nullptr;
    float x[RT * RT];
    bool on[RT * RT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < RT; j++) {
            const int wa = a0 + ty * RT + i, wb = b0 + tx + 16 * j, u = RT * i + j;
            x[u] = acc[i][j];
            on[u] = wa < a.W && wb < wa;
            if (on[u] && (!(x[u] == x[u]) || isinf(x[u]))) {
                any_nan = true;
                on[u] = false;
            }
            if (on[u] && a.fcd) a.fcd[(size_t)sim * a.n_fcd + (size_t)wa * (wa - 1) / 2 + wb] = x[u];
        }
    if (hist) ks_count<RT * RT>(a.emp_sorted, a.ks_lut, a.m, x, on, hist, eq);
    if (any_nan && a.nan_flag) atomicOr(&a.nan_flag[sim], 1);
}

// ------------------------------------------------------------ KS + GOF

__device__ double block_sum(double v, double* sh) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w];
    return s;
}

__device__ double block_max(double v, double* sh) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s = fmax(s, sh[w]);
    return s;
}

// One cluster of CTAs per simulation; every CTA takes a share of the KS bins
// and every warp a contiguous piece of that, so the bins are read in whole
// lines (one thread per contiguous piece of one CTA's bins read them 4 bytes
// at a time at a stride of kilobytes: 0.90 ms for 4 simulations of 668,746
// bins, 0.20 ms for 64 of 146,070; now 0.12 and 0.09 ms).  Rank 0 does the FC and the cost.
__global__ void __launch_bounds__(1024) gof_kernel(GofArgs a) {
    __shared__ double sh[32];
    __shared__ unsigned int wtot[32], total;  // FCD values counted in each warp's bins, in this CTA's
    __shared__ double dks[8];                 // rank 0: every CTA's KS distance
    const int rank = (int)cluster_rank(), ranks = (int)cluster_size();
    const int sim = blockIdx.x / ranks, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!a.no_fcd) {
        // KS: D = max over jump points c of |c/m - F_sim| just before/at the point
        const int nb = a.m + 1, nw = ranks * 32;
        const unsigned int* h = a.hist + (size_t)sim * nb;
        const unsigned int* q = a.eq + (size_t)sim * nb;
        const int per = ((nb + nw - 1) / nw + 31) / 32 * 32;
        const int c0 = min(nb, (rank * 32 + warp) * per), c1 = min(nb, c0 + per);
        unsigned int loc = 0;
#pragma unroll 4
        for (int c = c0 + lane; c < c1; c += 32) loc += h[c];
        loc = __reduce_add_sync(0xffffffffu, loc);
        if (lane == 0) wtot[warp] = loc;
        __syncthreads();
        unsigned int H = __reduce_add_sync(0xffffffffu, lane < warp ? wtot[lane] : 0u);  // sims with rank < c0
        if (threadIdx.x == 0) {
            unsigned int t = 0;
            for (int w = 0; w < 32; w++) t += wtot[w];
            total = t;
        }
        __syncwarp();  // the cluster barrier is warp-wide (.aligned)
        cluster_sync();
        for (int r = 0; r < rank; r++) H += ld_cluster_u32(map_rank(smem_u32(&total), (uint32_t)r));
        const double invm = 1.0 / a.m, invn = 1.0 / a.n_fcd;
        double dmax = 0.0;
        constexpr int U = 4;  // lines of 32 bins in flight
        for (int b = c0; b < c1; b += 32 * U) {
            unsigned int hv[U], qv[U], inc[U];
            bool ok[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int c = b + 32 * u + lane;
                const bool in = c < c1;
                hv[u] = in ? h[c] : 0u;
                qv[u] = in ? q[c] : 0u;
                ok[u] = in && a.valid[c];
                inc[u] = hv[u];
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const unsigned int v = __shfl_up_sync(0xffffffffu, inc[u], o);
                    if (lane >= o) inc[u] += v;
                }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const unsigned int Hc = H + inc[u] - hv[u];  // sims with rank < c
                const double Fe = (b + 32 * u + lane) * invm;
                if (ok[u]) {
                    dmax = fmax(dmax, fabs(Fe - (double)(Hc + qv[u]) * invn));
                    dmax = fmax(dmax, fabs(Fe - (double)(Hc + hv[u]) * invn));
                }
                H += __shfl_sync(0xffffffffu, inc[u], 31);
            }
        }
        const double D = block_max(dmax, sh);
        if (threadIdx.x == 0) st_cluster_f64(map_rank(smem_u32(&dks[rank]), 0), D);
    }
    // also keeps every CTA's total in place until all have read it
    __syncwarp();
    cluster_sync();
    if (rank != 0) return;
    double D = 0.0;
    if (!a.no_fcd)
        for (int r = 0; r < ranks; r++) D = fmax(D, dks[r]);
    // FC: Pearson with the empirical FC, and mean difference (FP64, two passes)
    const float* fc = a.fc + (size_t)sim * a.P;
    double s = 0.0;
    for (int p = threadIdx.x; p < a.P; p += blockDim.x) s += fc[p];
    const double msim = block_sum(s, sh) / a.P;
    double sxy = 0, sxx = 0, syy = 0;
    for (int p = threadIdx.x; p < a.P; p += blockDim.x) {
        const double dx = a.emp_fc[p] - a.emp_fc_mean, dy = (double)fc[p] - msim;
        sxy += dx * dy;
        sxx += dx * dx;
        syy += dy * dy;
    }
    sxy = block_sum(sxy, sh);
    sxx = block_sum(sxx, sh);
    syy = block_sum(syy, sh);
    const double r = sxy / (sqrt(sxx) * sqrt(syy));
    double pen = 0.0;
    if (a.calc_fic_penalty) {
        double ps = 0.0;
        for (int j = threadIdx.x; j < a.N; j += blockDim.x) {
            const double d = fabs(a.ext[((size_t)sim * 6 + 2) * a.N + j] - 3);
            if (d > 1) ps += 1 - exp(-0.05 * (d - 1));
        }
        pen = block_sum(ps, sh) * a.fic_penalty_scale / a.N;
        if (a.fic_reject_failed && a.failed[sim]) pen += 1;
    }
    if (threadIdx.x == 0) {
        const double diff = fabs(a.emp_fc_mean - msim);
        double c = 1 - r + (a.use_fc_diff ? diff : 0.0) + D;
        const bool bad = a.nan_flag[sim] != 0 || !(r == r);
        if (bad) c = a.max_cost;
        a.cost[sim] = c;
        a.fc_corr[sim] = r;
        a.fc_diff[sim] = diff;
        a.fcd_ks[sim] = D;
        a.fic_penalty[sim] = a.calc_fic_penalty ? pen : 0.0;
    }
}

}  // namespace bnm

using namespace bnm;

template <typename TB, int RI, int RJ>
static cudaError_t launch_fc_window_t(const FcArgs& a, const TB* bold, cudaStream_t st) {
    constexpr int TI = 16 * RI, TJ = 16 * RJ, NT = TI + TJ, threads = 256 + (RI + RJ + 1) / 2 * 32;
    // window lengths are limited by what a ring of all nodes would take of one SM
    if ((size_t)a.N * 5 * sizeof(double) + (size_t)a.win_len * a.N * sizeof(TB) > 227 * 1024) return cudaErrorInvalidValue;
    const int M = a.exc ? a.N / 2 : a.N;
    int tiles = 0;  // as the kernel counts them
    for (int bi = 0; bi * TI < M; bi++) {
        const int imax = std::min((bi + 1) * TI, M) - 1;
        tiles += imax < 1 ? 0 : (imax - 1) / TJ + 1;
    }
    if (a.exc) tiles *= 2;
    if (tiles < 1) return cudaErrorInvalidValue;
    // the ring holds the window and two chunks where that leaves room for two
    // CTAs an SM; else two chunks, and the frames that leave a window are read again
    const size_t fixed = (size_t)2 * kChunk * NT * sizeof(double2) + NT * (sizeof(double2) + sizeof(double)) +
                         2 * (kChunk + 1) * sizeof(int);
    const int full = a.win_len + 2 * kChunk;
    const bool ring = (size_t)full * NT * sizeof(double) + fixed <= 110 * 1024;
    const int rl = ring ? full : 2 * kChunk;
    const size_t smem = (size_t)rl * NT * sizeof(double) + fixed;
    auto* fn = ring ? fc_window_kernel<TB, RI, RJ, true> : fc_window_kernel<TB, RI, RJ, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    fn<<<dim3(a.n_sims, tiles), threads, smem, st>>>(a, bold, rl);
    return cudaGetLastError();
}

// The window tile: each CTA of 256 pair threads carries 256 ppt pairs (nodes
// 16 x 16, 16 x 32, 32 x 32 or 32 x 64) through the frames; fewer pairs per
// CTA give more CTAs but repeat the nodes' series per CTA.  The plan's tuner
// picks ppt; without one, the largest tile that still gives two CTAs an SM.
template <typename TB>
static cudaError_t launch_fc_window(const FcArgs& a, const TB* bold, cudaStream_t st) {
    int ppt = a.ppt;
    if (!ppt) {
        // of the smallest tile; 300: two for each of the GPU's 148 SMs
        const long long ctas = (long long)a.P * a.n_sims / 256;
        ppt = ctas >= 8 * 300 ? 8 : ctas >= 4 * 300 ? 4 : ctas >= 2 * 300 ? 2 : 1;
    }
    switch (ppt) {
        case 1: return launch_fc_window_t<TB, 1, 1>(a, bold, st);
        case 2: return launch_fc_window_t<TB, 1, 2>(a, bold, st);
        case 4: return launch_fc_window_t<TB, 2, 2>(a, bold, st);
        case 8: return launch_fc_window_t<TB, 2, 4>(a, bold, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t bnm_launch_fc_window(const FcArgs& a, cudaStream_t st) {
    if (a.W >= 1 && a.P < 2) return cudaErrorInvalidValue;  // a window row of one value cannot be centred
    return a.bold_f64 ? launch_fc_window<double>(a, a.bold_f64, st) : launch_fc_window<float>(a, a.bold, st);
}

// Window-FC sums over a pair range, one CTA per (window, simulation): the
// centring of fcd_gram_kernel's FCDs, over all pairs or (window_fc_stats with
// save_hemis, bnm.cu:436-496) a hemisphere's.
__global__ void __launch_bounds__(256) window_sums_kernel(const float* wfc, int W, int P, int p0, int p1,
                                                          double* out) {
    __shared__ double sh[16];
    const int w = blockIdx.x, sim = blockIdx.y;
    double ws[2];
    window_sums(wfc + ((size_t)sim * W + w) * P, p0, p1, sh, ws);
    if (threadIdx.x == 0) {
        out[((size_t)sim * W + w) * 2] = ws[0];
        out[((size_t)sim * W + w) * 2 + 1] = ws[1];
    }
}

cudaError_t bnm_launch_window_sums(const float* wfc, int n_sims, int W, int P, int p0, int p1, double* wsum_out,
                                   cudaStream_t st) {
    if (p0 < 0 || p1 > P || p1 - p0 < 2) return cudaErrorInvalidValue;
    window_sums_kernel<<<dim3(W, n_sims), 256, 0, st>>>(wfc, W, P, p0, p1, wsum_out);
    return cudaGetLastError();
}

cudaError_t bnm_launch_fcd(const FcdArgs& a, cudaStream_t st) {
    auto tiles = [&](int tile) {
        const int side = (a.W + tile - 1) / tile;
        return side * (side + 1) / 2;
    };
    // The larger tile reads each row half as often and costs 2.5-2.8 of the
    // smaller: it pays where there are two CTAs of it for each SM (296) and the
    // windows do not leave much of it empty (W = 278, 15 tiles against 45, 64
    // simulations: 0.92 against 1.04 ms; W = 85, 3 against 6, 300 simulations:
    // 132 against 110 us; 60 tiles in all: 169 against 116 us).
    if ((long long)tiles(64) * a.n_sims >= 296 && 8 * tiles(64) < 3 * tiles(32))
        fcd_gram_kernel<64><<<dim3(tiles(64), a.n_sims), 256, 0, st>>>(a);
    else
        fcd_gram_kernel<32><<<dim3(tiles(32), a.n_sims), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t bnm_launch_gof(const GofArgs& a, cudaStream_t st) {
    // 8 CTAs a simulation where the bins are many; a small histogram (a warp
    // then has fewer than four lines) is one CTA's
    const int ranks = a.no_fcd || a.m < 4096 ? 1 : 8;
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(a.n_sims * ranks));
    cfg.blockDim = dim3(1024);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, gof_kernel, a);
}
