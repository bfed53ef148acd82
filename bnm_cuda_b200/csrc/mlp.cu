// MLP surrogate of the simulate-and-fit cost (no counterpart in the
// reference): maps (G, wEE, wEI, SC spectral summary) to the fit terms so that
// oversampled CMA-ES candidates can be pre-screened before simulation.
//
// Network: in -> [hidden, ReLU] x layers -> out, weights kept in FP32 (master
// copy for Adam) and rounded to BF16 for the GEMMs; activations are stored in
// BF16; every GEMM accumulates in FP32 (mma.sync m16n8k16).  Training (MSE
// loss, Adam) runs entirely on the device.
//
//   mlp_step_kernel     any number of training steps (forward, loss, backward,
//                       Adam) in one launch of one thread-block cluster; also
//                       one step's loss and gradients, and the forward pass of
//                       networks too wide for the kernel below
//   mlp_predict_kernel  forward pass, 16 rows per CTA, activations in shared
//                       memory
//
// A step of the surrogate is small (B = 64, 256 wide: 78 MFLOP) and a chain of
// 2 L dependent GEMMs, so it is bound by latency: of launches, of the loads in
// front of each GEMM and of the K loop.  One kernel per GEMM took 574 us a step
// (24 launches, GEMM grids of 4 CTAs at 12-108 us each: one 64 x 64 tile per
// CTA, element-wise strided loads and two block barriers per 32 K).  Here the
// phases of a step are separated by the cluster's hardware barrier, and every
// operand is kept in the order in which the MMA's lanes hold it, in both
// orientations where two GEMMs need it, padded with zeros to multiples of 16:
//   A blocks  16 rows x 16 K as uint4 [lane]   (the four A registers)
//   B blocks   8 rows x 16 K as uint2 [lane]   (the two B registers)
// so a K step of a 16 x 8 output tile is one 16-byte and one 8-byte coalesced
// load per lane (as rows, the same step touched eight cache lines a load:
// 145 us a step), all K steps of a 256-wide layer are in flight at once, a
// warp's tiles come in twos that share an operand (one tile at a time behind a
// function call: 100 us a step), and an epilogue writes the next
// GEMM's operand from its accumulators' own lanes, transposed by movmatrix
// where the other orientation is wanted.  FP32 weights and Adam's moments are
// kept in accumulator order too ([tile][lane] float4), and Adam runs in the
// epilogue of the dW tiles; a layer's weights are updated one phase after the
// last GEMM that reads them.  The K order of every output's MMAs is ascending
// in steps of 16 and the other sums are in index order, whatever the cluster
// size and the tiling.  Measured (19-4x256-4, 2000 rows, batch 64, 4 epochs,
// parameters set and read back): 71.3 -> 6.2 ms; about 40 us of a step's 42
// are its 10 phases' load and barrier latencies and Adam.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>

#include "../../include/bnm_b200.h"
#include "cluster_util.cuh"
#include "kernels.h"

int bnm_fail_cuda(cudaError_t e, const char* expr, const char* file, int line);
int bnm_fail_msg(int code, const char* msg);

namespace {

using bnm::cluster_rank;
using bnm::cluster_size;
using bnm::cluster_sync;
typedef __nv_bfloat16 bf16;

// A layer on the device.  dinp, doutp: din, dout rounded up to 16.
struct MlpLayer {
    int din, dout, dinp, doutp;
    long long woff, boff;  // W and b in the caller's flat parameter vector
    long long tile, bias;  // W's tiles (16 o x 8 i; units of one tile) and b in the device's FP32 arrays
    uint2 *w, *wt;         // BF16 weights as B blocks: n = output, k = input; and n = input, k = output
    uint4* x;              // input activations as A blocks, k = input (first layer: two sets, by step parity)
    uint2* xt;             // ... as B blocks, n = input, k = batch row (likewise)
    float* dz;             // gradient at the layer's output, behind its ReLU mask [batch][doutp]
    uint4 *dzh, *dzt;      // the same rounded, as A blocks: k = output; and m = output, k = batch row
};

enum { kTrain = 0, kGrads = 1, kForward = 2 };

struct StepArgs {
    const MlpLayer* layers;
    int L, in, out;
    int mode, steps, batch;
    float4 *w, *m, *v;     // weights and Adam moments, [tile][lane] in accumulator order
    float *bw, *bm, *bv;   // biases
    float* g;              // flat gradient (kGrads)
    const float *X, *T;    // [.][in], [.][out]
    const int* idx;        // [steps][batch] rows of X and T, or null: row b
    const float2* c12;     // [steps] Adam bias corrections
    float lr, b1, b2, eps;
    size_t x0, xt0;        // elements of one set of the first layer's x and xt
    float* tgt;            // [2][batch][out]: targets of the step's rows, by step parity
    float *yout, *loss;    // [batch][out]; [steps]
};

__device__ __forceinline__ uint32_t pack2(float x, float y) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x)) |
           ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(y)) << 16);
}

// The matrix instructions below are warp-wide (.aligned): all 32 lanes execute
// them together.  A branch that only some lanes take (rows past the batch,
// columns past a layer, Adam's plain expression) is followed by __syncwarp()
// before the next of them.

// 8 x 8 BF16 transpose across the warp: lane (g, t) holds row g, columns 2t, 2t + 1
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint4& a, const uint2& b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y));
}

// Output tiles of 16 x 8: kb MMAs each in ascending K, kFly K blocks in flight
// ahead of their MMAs (the rest of kb in halving groups, so that no load is
// predicated).  load(k, a, b): this lane's registers of K block k, nA A blocks
// times nB B blocks.
template <int kFly, int nA, int nB, class F>
__device__ __forceinline__ void mma_group(int k0, float (&d)[nA * nB][4], F load) {
    uint4 a[kFly][nA];
    uint2 b[kFly][nB];
#pragma unroll
    for (int s = 0; s < kFly; s++) load(k0 + s, a[s], b[s]);
#pragma unroll
    for (int s = 0; s < kFly; s++)
#pragma unroll
        for (int i = 0; i < nA * nB; i++) mma_bf16(d[i], a[s][i / nB], b[s][i % nB]);
}
template <int kFly, int nA, int nB, class F>
__device__ __forceinline__ void mma_rest(int k0, int kb, float (&d)[nA * nB][4], F load) {
    if (k0 + kFly <= kb) {
        mma_group<kFly, nA, nB>(k0, d, load);
        k0 += kFly;
    }
    if constexpr (kFly > 1) mma_rest<kFly / 2, nA, nB>(k0, kb, d, load);
}
template <int kFly, int nA, int nB, class F>
__device__ __forceinline__ void mma_tiles(int kb, float (&d)[nA * nB][4], F load) {
#pragma unroll
    for (int i = 0; i < nA * nB; i++) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
    __syncwarp();
    int k0 = 0;
#pragma unroll 1
    for (; k0 + kFly <= kb; k0 += kFly) mma_group<kFly, nA, nB>(k0, d, load);
    if constexpr (kFly > 1) mma_rest<kFly / 2, nA, nB>(k0, kb, d, load);
}

// Adam's update of nP parameters (w, first moment m, second moment v; g the
// gradients).  The update is the FP32 expression
//     w - lr (m / c1) / (sqrt(v / c2) + eps)
// with every operation rounded to nearest.  The hardware has no FP32 division
// or square root: CUDA's are subroutines with a branch each, which a warp goes
// through one after the other (about 6000 cycles for the 8 parameters of a
// lane).  Here the quotients and the root are formed in FP64, without branches,
// so the parameters' chains interleave, and rounded to FP32.  That gives the
// same FP32 values: a quotient of two 24-bit numbers is at least 2^-49 away
// (relative) from the midpoint of two FP32 neighbours, and the root of one at
// least 2^-51 (x - y^2, for a midpoint y, is an odd multiple of 2^-48 with x in
// [1, 4), hence |sqrt(x) - y| / y > 2^-49 / x), unless the result is subnormal.
// The FP64 errors are below that: two roundings, 2^-52, for the quotients by
// rc1, rc2; the last step's rounding, 2^-53, plus what the Newton steps leave of
// the 2^-22 estimates (less than 2^-60 for the root, 2^-88 for the quotient).
// Lanes with a value near the ends of the range take the plain expression.
__device__ __forceinline__ float adam_plain(float w, float m, float v, const StepArgs& a, float c1, float c2) {
    return w - a.lr * (m / c1) / (sqrtf(v / c2) + a.eps);
}
template <int nP>
__device__ __forceinline__ void adam(const float (&g)[nP], float (&w)[nP], float (&m)[nP], float (&v)[nP],
                                     const StepArgs& a, float2 c12, double rc1, double rc2) {
    float nw[nP];
    bool ok = true;
    auto safe = [](float x, float lo) { return x == 0.f || (fabsf(x) > lo && fabsf(x) < 1e27f); };
#pragma unroll
    for (int i = 0; i < nP; i++) {
        m[i] = fmaf(1.f - a.b1, g[i], a.b1 * m[i]);
        v[i] = fmaf((1.f - a.b2) * g[i], g[i], a.b2 * v[i]);
        const float mh = (float)((double)m[i] * rc1), vh = (float)((double)v[i] * rc2);
        // root: two Newton steps on g ~ sqrt(x) with the slope of the first estimate
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(vh));
        const double x = vh, h = 0.5 * (double)y;
        double r = x * (double)y;
        r = fma(fma(-r, r, x), h, r);
        r = fma(fma(-r, r, x), h, r);
        const float den = (vh == 0.f ? 0.f : (float)r) + a.eps, num = a.lr * mh;
        // quotient: one Newton step on the reciprocal, one on the quotient
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(den));
        const double d = den, nd = num;
        double q = y;
        q = fma(fma(-d, q, 1.0), q, q);
        const double q0 = nd * q;
        nw[i] = w[i] - (float)fma(fma(-d, q0, nd), q, q0);
        ok = ok && safe(m[i], 1e-27f) && safe(v[i], 1e-27f) && safe(num, 1e-18f) && den > 1e-18f && den < 1e18f;
    }
    if (!ok)
#pragma unroll
        for (int i = 0; i < nP; i++) nw[i] = adam_plain(w[i], m[i], v[i], a, c12.x, c12.y);
#pragma unroll
    for (int i = 0; i < nP; i++) w[i] = nw[i];
}

constexpr int kStepThreads = 512, kStepWarps = kStepThreads / 32;
constexpr int kPredThreads = 512, kPredWarps = kPredThreads / 32;
constexpr int kSmemLayers = 128;  // layer descriptors kept in shared memory (more are read from L1)

// What a step's tile functions share.
struct Step {
    const StepArgs& a;
    const MlpLayer* lay;
    int par;         // step parity
    float2 c12;
    double rc1, rc2; // reciprocals of c12
    int mt;          // blocks of 16 batch rows

    __device__ const uint4* x(int l) const { return lay[l].x + (l == 0 && par ? a.x0 : 0); }
    __device__ const uint2* xt(int l) const { return lay[l].xt + (l == 0 && par ? a.xt0 : 0); }
    __device__ float* tgt() const { return a.tgt + (size_t)par * a.batch * a.out; }
};

// The rows of X that step `step` uses, rounded, as the first layer's operands
// (block mb of 16 rows, block k of 16 columns); and their targets (32 values a
// task).  Done while the step before ends: the gathers are chains of loads.
__device__ __forceinline__ void gather_x(const Step& st, int step, int mb, int k) {
    const StepArgs& a = st.a;
    const int lane = threadIdx.x & 31, c = 16 * k + 2 * (lane & 3), B = a.batch, kb = st.lay[0].dinp / 16;
    uint32_t v[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int m = 16 * mb + (lane >> 2) + 8 * h;
        const float* p = m < B ? a.X + (size_t)(a.idx ? a.idx[(size_t)step * B + m] : m) * a.in : nullptr;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = c + 8 * q;
            v[h + 2 * q] = pack2(p && i < a.in ? p[i] : 0.f, p && i + 1 < a.in ? p[i + 1] : 0.f);
        }
    }
    uint4* x = st.lay[0].x + (step & 1 ? a.x0 : 0);
    uint2* xt = st.lay[0].xt + (step & 1 ? a.xt0 : 0) + lane;
    x[(size_t)(mb * kb + k) * 32 + lane] = make_uint4(v[0], v[1], v[2], v[3]);
    __syncwarp();
    xt[(size_t)(2 * k * st.mt + mb) * 32] = make_uint2(transpose8(v[0]), transpose8(v[1]));
    xt[(size_t)((2 * k + 1) * st.mt + mb) * 32] = make_uint2(transpose8(v[2]), transpose8(v[3]));
}
__device__ __forceinline__ void gather_t(const StepArgs& a, int step, int task) {
    const int e = 32 * task + (threadIdx.x & 31), n = a.batch * a.out;
    if (e >= n) return;
    const int b = e / a.out;
    const int r = a.idx ? a.idx[(size_t)step * a.batch + b] : b;
    a.tgt[(size_t)(step & 1) * n + e] = a.T[(size_t)r * a.out + e % a.out];
}

// Writes the gradient e of a 16 x 8 tile (rows 16 mb .., columns 8 nb ..) at
// the output of layer z: FP32, and rounded in both orientations.
__device__ __forceinline__ void store_dz(const Step& st, const MlpLayer& z, int mb, int nb, const float (&e)[4]) {
    const int lane = threadIdx.x & 31, m = 16 * mb + (lane >> 2), n = 8 * nb + 2 * (lane & 3), B = st.a.batch;
    if (m < B) *reinterpret_cast<float2*>(z.dz + (size_t)m * z.doutp + n) = make_float2(e[0], e[1]);
    if (m + 8 < B) *reinterpret_cast<float2*>(z.dz + (size_t)(m + 8) * z.doutp + n) = make_float2(e[2], e[3]);
    const uint32_t p0 = pack2(e[0], e[1]), p1 = pack2(e[2], e[3]);
    // columns 8 nb .. are registers 0, 1 or 2, 3 of A block nb / 2
    reinterpret_cast<uint2*>(z.dzh + ((size_t)mb * (z.doutp / 16) + nb / 2) * 32 + lane)[nb & 1] = make_uint2(p0, p1);
    uint32_t* zt = reinterpret_cast<uint32_t*>(z.dzt + ((size_t)(nb / 2) * st.mt + mb) * 32 + lane) + (nb & 1);
    __syncwarp();
    zt[0] = transpose8(p0);
    zt[2] = transpose8(p1);
}

// Forward of layer l, 8 outputs of nA blocks of 16 rows; the last layer also
// forms the gradient of the MSE at its output.
template <int nA>
__device__ __forceinline__ void forward_tiles(const Step& st, int l, int mb, int nb) {
    const StepArgs& a = st.a;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, B = a.batch;
    const MlpLayer& y = st.lay[l];
    const int n = 8 * nb + 2 * t, kb = y.dinp / 16;
    const float2 bias = *reinterpret_cast<const float2*>(a.bw + y.bias + n);
    const uint2* wp = y.w + (size_t)nb * kb * 32 + lane;
    const uint4* xp = st.x(l) + (size_t)mb * kb * 32 + lane;
    float d[nA][4];
    mma_tiles<8, nA, 1>(kb, d, [&](int k, uint4 (&fa)[nA], uint2 (&fb)[1]) {
#pragma unroll
        for (int i = 0; i < nA; i++) fa[i] = xp[32 * (i * kb + k)];
        fb[0] = wp[32 * k];
    });
#pragma unroll
    for (int i = 0; i < nA; i++) {
        const int m = 16 * (mb + i) + g;
        const float v[4] = {d[i][0] + bias.x, d[i][1] + bias.y, d[i][2] + bias.x, d[i][3] + bias.y};
        if (l < a.L - 1) {  // rows past the batch and columns past the layer are zero
            const MlpLayer& z = st.lay[l + 1];
            const uint32_t p0 = m < B ? pack2(fmaxf(v[0], 0.f), fmaxf(v[1], 0.f)) : 0u;
            const uint32_t p1 = m + 8 < B ? pack2(fmaxf(v[2], 0.f), fmaxf(v[3], 0.f)) : 0u;
            reinterpret_cast<uint2*>(z.x + ((size_t)(mb + i) * (z.dinp / 16) + nb / 2) * 32 + lane)[nb & 1] =
                make_uint2(p0, p1);
            __syncwarp();
            if (a.mode != kForward)
                z.xt[((size_t)nb * st.mt + mb + i) * 32 + lane] = make_uint2(transpose8(p0), transpose8(p1));
            continue;
        }
        float e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = m + 8 * (q >> 1), c = n + (q & 1);
            e[q] = 0.f;
            if (r < B && c < a.out) {
                a.yout[(size_t)r * a.out + c] = v[q];
                if (a.mode != kForward) {  // MSE: d loss / dy = 2 (y - t) / (B out)
                    const float df = v[q] - st.tgt()[(size_t)r * a.out + c];
                    e[q] = 2.f * df / (float)(B * a.out);
                }
            }
        }
        if (a.mode != kForward) store_dz(st, y, mb + i, nb, e);
    }
}

// dX of layer l, 8 inputs of nA blocks of 16 rows: the gradient at the output
// of layer l - 1, behind its ReLU.
template <int nA>
__device__ __forceinline__ void dx_tiles(const Step& st, int l, int mb, int nb) {
    const int lane = threadIdx.x & 31;
    const MlpLayer& y = st.lay[l];
    const int kb = y.doutp / 16;
    const uint4* ap = y.dzh + (size_t)mb * kb * 32 + lane;
    const uint2* bp = y.wt + (size_t)nb * kb * 32 + lane;
    // the activations behind the mask sit in this lane's own registers of the A block
    uint2 act[nA];
#pragma unroll
    for (int i = 0; i < nA; i++)
        act[i] = reinterpret_cast<const uint2*>(st.x(l) + ((size_t)(mb + i) * (y.dinp / 16) + nb / 2) * 32 + lane)[nb & 1];
    float d[nA][4];
    mma_tiles<8, nA, 1>(kb, d, [&](int k, uint4 (&fa)[nA], uint2 (&fb)[1]) {
#pragma unroll
        for (int i = 0; i < nA; i++) fa[i] = ap[32 * (i * kb + k)];
        fb[0] = bp[32 * k];
    });
#pragma unroll
    for (int i = 0; i < nA; i++) {
        float e[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t xb = q < 2 ? act[i].x : act[i].y;
            const float x = __uint_as_float((q & 1) ? xb & 0xffff0000u : xb << 16);
            e[q] = x > 0.f ? d[i][q] : 0.f;  // rows past the batch have x = 0
        }
        store_dz(st, st.lay[l - 1], mb + i, nb, e);
    }
}

// Bias gradients of 32 outputs: sums over the batch in order.
__device__ __forceinline__ void db_task(const Step& st, int l, int task) {
    const StepArgs& a = st.a;
    const MlpLayer& y = st.lay[l];
    const int o = task * 32 + (threadIdx.x & 31), B = a.batch, ld = y.doutp;
    if (o >= y.dout) return;
    const float* dz = y.dz + o;
    float s = 0.f;
    int b = 0;
    for (; b + 16 <= B; b += 16) {
        float e[16];
#pragma unroll
        for (int k = 0; k < 16; k++) e[k] = dz[(size_t)(b + k) * ld];
#pragma unroll
        for (int k = 0; k < 16; k++) s += e[k];
    }
    for (; b < B; b++) s += dz[(size_t)b * ld];
    if (a.mode == kGrads) {
        a.g[y.boff + o] = s;
        return;
    }
    const long long i = y.bias + o;
    float gi[1] = {s}, wi[1] = {a.bw[i]}, mi[1] = {a.bm[i]}, vi[1] = {a.bv[i]};
    adam(gi, wi, mi, vi, a, st.c12, st.rc1, st.rc2);
    a.bm[i] = mi[0];
    a.bv[i] = vi[0];
    a.bw[i] = wi[0];
}

// dW of layer l, 16 outputs o x 16 inputs i (two tiles), K = batch, and Adam's
// update of its weights; the tasks past the tiles are the biases'.
__device__ __forceinline__ void dw_task(const Step& st, int l, int task) {
    const StepArgs& a = st.a;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const MlpLayer& y = st.lay[l];
    const int ot = y.doutp / 16, ki = y.dinp / 16;
    if (task >= ot * ki) {
        db_task(st, l, task - ot * ki);
        return;
    }
    const int ob = task % ot, ib = 2 * (task / ot), kb = st.mt;
    const bool train = a.mode == kTrain;
    const size_t e = (size_t)(y.tile + ib * ot + ob) * 32 + lane;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 wv[2], mv[2], vv[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {  // the parameters' loads overlap the MMAs
        const size_t ei = e + (size_t)i * ot * 32;
        wv[i] = train ? a.w[ei] : zero;
        mv[i] = train ? a.m[ei] : zero;
        vv[i] = train ? a.v[ei] : zero;
    }
    const uint4* ap = y.dzt + (size_t)ob * kb * 32 + lane;
    float d[2][4];
    const uint2* bp = st.xt(l) + (size_t)ib * kb * 32 + lane;
    mma_tiles<4, 1, 2>(kb, d, [&](int k, uint4 (&fa)[1], uint2 (&fb)[2]) {
        fa[0] = ap[32 * k];
        fb[0] = bp[32 * k];
        fb[1] = bp[32 * (kb + k)];
    });
    auto inside = [&](int i, int q) {  // accumulator q of tile i is a weight, not padding
        return 16 * ob + g + 8 * (q >> 1) < y.dout && 8 * (ib + i) + 2 * t + (q & 1) < y.din;
    };
    if (!train) {
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int i = k >> 2, q = k & 3, o = 16 * ob + g + 8 * (q >> 1), c = 8 * (ib + i) + 2 * t + (q & 1);
            if (inside(i, q)) a.g[y.woff + (long long)o * y.din + c] = d[i][q];
        }
        return;
    }
    const float gr[8] = {d[0][0], d[0][1], d[0][2], d[0][3], d[1][0], d[1][1], d[1][2], d[1][3]};
    float w[8] = {wv[0].x, wv[0].y, wv[0].z, wv[0].w, wv[1].x, wv[1].y, wv[1].z, wv[1].w};
    float m[8] = {mv[0].x, mv[0].y, mv[0].z, mv[0].w, mv[1].x, mv[1].y, mv[1].z, mv[1].w};
    float v[8] = {vv[0].x, vv[0].y, vv[0].z, vv[0].w, vv[1].x, vv[1].y, vv[1].z, vv[1].w};
    adam(gr, w, m, v, a, st.c12, st.rc1, st.rc2);
#pragma unroll
    for (int i = 0; i < 2; i++) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (!inside(i, q)) w[4 * i + q] = m[4 * i + q] = v[4 * i + q] = 0.f;  // the padding stays zero
        __syncwarp();
        const size_t ei = e + (size_t)i * ot * 32;
        a.w[ei] = make_float4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        a.m[ei] = make_float4(m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]);
        a.v[ei] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        const uint32_t p0 = pack2(w[4 * i], w[4 * i + 1]), p1 = pack2(w[4 * i + 2], w[4 * i + 3]);
        uint32_t* wp = reinterpret_cast<uint32_t*>(y.w + ((size_t)(2 * ob) * ki + ib / 2) * 32 + lane) + i;
        wp[0] = p0;
        wp[(size_t)ki * 64] = p1;  // the next 8 outputs' block
        y.wt[((size_t)(ib + i) * ot + ob) * 32 + lane] = make_uint2(transpose8(p0), transpose8(p1));
    }
}

// One cluster; CTA c of it takes the c-th share of a phase's tiles, a warp per
// tile.  A forward pass alone may have several clusters: they take blocks of
// rows of their own, and none waits for another (one cluster for all rows took
// 26 ms for 8192 rows of 19-3x4096-4 where a launch per GEMM had taken 22; now
// 7.7).  Phases of a step, each ending in a cluster barrier:
//   forward of layer 0 .. L-1 (the last also forms the output gradient);
//   for l = L-1 .. 1: dX of layer l, with dW / db (and Adam) of layer l + 1;
//   dW / db of layers 1 and 0, and the next step's rows of X and T.
__global__ void __launch_bounds__(kStepThreads, 1) mlp_step_kernel(StepArgs args) {
    __shared__ float red[256];
    __shared__ MlpLayer s_lay[kSmemLayers];
    const int warp = threadIdx.x >> 5;
    const int nc = (int)cluster_size(), c = (int)cluster_rank();
    const int L = args.L, B = args.batch;
    if (L <= kSmemLayers)
        for (int e = threadIdx.x; e < L * (int)sizeof(MlpLayer) / 4; e += kStepThreads)
            reinterpret_cast<uint32_t*>(s_lay)[e] = reinterpret_cast<const uint32_t*>(args.layers)[e];
    __syncthreads();
    const MlpLayer* lay = L <= kSmemLayers ? s_lay : args.layers;
    // blocks of 16 rows, taken in twos; this cluster's: mg twos from block mb0
    const int mt = (B + 15) / 16, twos = (mt + 1) / 2;
    const int clusters = gridDim.x / nc, per = (twos + clusters - 1) / clusters;
    const int mb0 = 2 * min(twos, (int)(blockIdx.x / nc) * per), mg = min(twos, mb0 / 2 + per) - mb0 / 2;
    Step st{args, lay, 0, make_float2(1.f, 1.f), 1.0, 1.0, mt};

    // this CTA's shares of up to three task lists, dealt to its warps.  Every
    // list is shared out by itself: as one, gathers and weight tiles of the last
    // phase fell to different CTAs, and with many inputs one CTA had all tiles
    // (4096 inputs, 256 wide, batch 4096: 11.5 ms a step, now 1.9)
    auto for_tasks = [&](int n1, int n2, int n3, auto&& f1, auto&& f2, auto&& f3) {
        const int p1 = (n1 + nc - 1) / nc, p2 = (n2 + nc - 1) / nc, p3 = (n3 + nc - 1) / nc;
        const int s1 = min(n1, c * p1), s2 = min(n2, c * p2), s3 = min(n3, c * p3);
        const int l1 = min(n1, s1 + p1) - s1, l2 = l1 + min(n2, s2 + p2) - s2, l3 = l2 + min(n3, s3 + p3) - s3;
        for (int k = warp; k < l3; k += kStepWarps) {
            if (k < l1)
                f1(s1 + k);
            else if (k < l2)
                f2(s2 + k - l1);
            else
                f3(s3 + k - l2);
            __syncwarp();
        }
        __syncwarp();
    };
    auto none = [](int) {};
    auto dw_tasks = [&](int l) { return (lay[l].doutp / 16) * (lay[l].dinp / 16) + (lay[l].dout + 31) / 32; };

    // gather tasks of a step: operand blocks, then targets
    const int kx = lay[0].dinp / 16, nx = (min(mt, mb0 + 2 * mg) - min(mt, mb0)) * kx, nt = args.mode == kForward ? 0 : (B * args.out + 31) / 32;
    auto gather = [&](int step, int task) {
        if (task < nx)
            gather_x(st, step, mb0 + task / kx, task % kx);
        else
            gather_t(args, step, task - nx);
    };
    for_tasks(nx + nt, 0, 0, [&](int task) { gather(0, task); }, none, none);
    cluster_sync();

    for (int step = 0; step < args.steps; step++) {
        st.par = step & 1;
        if (args.mode == kTrain) {
            st.c12 = args.c12[step];
            st.rc1 = 1.0 / (double)st.c12.x;
            st.rc2 = 1.0 / (double)st.c12.y;
        }

        for (int l = 0; l < L; l++) {
            for_tasks(mg * (lay[l].doutp / 8), 0, 0, [&](int task) {
                const int mb = mb0 + 2 * (task % mg), nb = task / mg;
                if (mb + 1 < mt)
                    forward_tiles<2>(st, l, mb, nb);
                else
                    forward_tiles<1>(st, l, mb, nb);
            }, none, none);
            cluster_sync();
        }
        if (args.mode == kForward) continue;

        // loss: mean over the batch of sum_o (y - t)^2 / out, by the last CTA
        if (c == nc - 1) {
            if (threadIdx.x < 256) {
                float s = 0.f;
                for (int i = threadIdx.x; i < B * args.out; i += 256) {
                    const float df = args.yout[i] - st.tgt()[i];
                    s += df * df;
                }
                red[threadIdx.x] = s;
            }
            __syncthreads();
            for (int k = 128; k; k >>= 1) {
                if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
                __syncthreads();
            }
            if (threadIdx.x == 0) args.loss[step] = red[0] / (float)(B * args.out);
        }
        for (int l = L - 1; l >= 1; l--) {
            for_tasks(mg * (lay[l].dinp / 8), l < L - 1 ? dw_tasks(l + 1) : 0, 0, [&](int task) {
                const int mb = 2 * (task % mg), nb = task / mg;
                if (mb + 1 < mt)
                    dx_tiles<2>(st, l, mb, nb);
                else
                    dx_tiles<1>(st, l, mb, nb);
            }, [&](int task) { dw_task(st, l + 1, task); }, none);
            cluster_sync();
        }
        // the last phase also gathers the next step's rows
        for_tasks(dw_tasks(1), step + 1 < args.steps ? nx + nt : 0, dw_tasks(0), [&](int task) { dw_task(st, 1, task); },
                  [&](int task) { gather(step + 1, task); }, [&](int task) { dw_task(st, 0, task); });
        cluster_sync();
    }
}

// Forward pass of 16 rows per CTA; the activations of two layers alternate in
// shared memory as A blocks.  X and Y may be page-locked host memory.  Rows are
// independent, so no CTA waits for another: 512 candidates on the 19-4x256-4
// network are 32 CTAs that each read the 410 KB of BF16 weights from L2.  A
// warp's tiles of all layers are one sequence whose weights do not depend on
// the activations, so they are copied ahead of their use (cp.async,
// kPredDepth tiles of the warp's own in shared memory), across the layers'
// barriers; each lane reads back what it copied.  The call at 512 rows: 48.7 us
// with loads at their use, which the compiler makes of every other form, 43.4
// copied ahead, 41.0 with X's loads all in flight as well.
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
constexpr int kPredDepth = 3;
template <bool kAhead>
__global__ void __launch_bounds__(kPredThreads) mlp_predict_kernel(const MlpLayer* layers, int L, int in, int out,
                                                                   int n, int width, const float* bw, const float* X,
                                                                   float* Y) {
    extern __shared__ __align__(16) uint4 sact[];  // [2][width / 16][32], then the warps' tiles of weights
    __shared__ MlpLayer s_lay[kSmemLayers];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * 16;
    if (L <= kSmemLayers)
        for (int e = threadIdx.x; e < L * (int)sizeof(MlpLayer) / 4; e += kPredThreads)
            reinterpret_cast<uint32_t*>(s_lay)[e] = reinterpret_cast<const uint32_t*>(layers)[e];
    __syncthreads();
    const MlpLayer* lay = L <= kSmemLayers ? s_lay : layers;
    const int tile = 2 * width;  // uint2 of a tile's weights (width / 16 blocks)
    uint2* const slots = reinterpret_cast<uint2*>(sact + 4 * width) + (size_t)warp * kPredDepth * tile + lane;
    int al = 0, an = warp, as = 0;  // the next tile to copy ahead (layer, block of outputs), its slot
    auto ahead = [&]() {
        while (al < L && an >= lay[al].doutp / 8) {
            al++;
            an = warp;
        }
        if (al < L) {
            const int kb = lay[al].dinp / 16;
            const uint2* src = lay[al].w + (size_t)an * kb * 32 + lane;
            uint2* dst = slots + (size_t)as * tile;
            for (int k = 0; k < kb; k++) cp_async8(dst + 32 * k, src + 32 * k);
            an += kPredWarps;
        }
        as = as + 1 == kPredDepth ? 0 : as + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (kAhead)
        for (int k = 0; k < kPredDepth - 1; k++) ahead();
    for (int k = warp; k < lay[0].dinp / 16; k += kPredWarps) {
        float v[8];  // all in flight at once: each is a trip to the host when X is there
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int r = r0 + g + 8 * (q >> 1 & 1), c = 16 * k + 2 * t + (q & 1) + 8 * (q >> 2);
            const float x = X[(size_t)min(r, n - 1) * in + min(c, in - 1)];
            v[q] = r < n && c < in ? x : 0.f;
        }
        sact[32 * k + lane] =
            make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    }
    __syncthreads();
    int slot = 0;
    for (int l = 0; l < L; l++) {
        const MlpLayer& y = lay[l];
        const int kb = y.dinp / 16;
        const uint4* src = sact + (l & 1) * 2 * width + lane;
        uint4* dst = sact + ((l + 1) & 1) * 2 * width + lane;
        for (int nb = warp; nb < y.doutp / 8; nb += kPredWarps) {
            const int c = 8 * nb + 2 * t;
            const float2 bias = *reinterpret_cast<const float2*>(bw + y.bias + c);
            float d[1][4];
            const uint2* wp;
            if (kAhead) {
                ahead();
                asm volatile("cp.async.wait_group %0;" ::"n"(kPredDepth - 1) : "memory");
                wp = slots + (size_t)slot * tile;
                slot = slot + 1 == kPredDepth ? 0 : slot + 1;
            } else {
                wp = y.w + (size_t)nb * kb * 32 + lane;
            }
            mma_tiles<8, 1, 1>(kb, d, [&](int k, uint4 (&fa)[1], uint2 (&fb)[1]) {
                fa[0] = src[32 * k];
                fb[0] = wp[32 * k];
            });
            const float v[4] = {d[0][0] + bias.x, d[0][1] + bias.y, d[0][2] + bias.x, d[0][3] + bias.y};
            if (l < L - 1) {
                reinterpret_cast<uint2*>(dst + 32 * (nb / 2))[nb & 1] = make_uint2(
                    pack2(fmaxf(v[0], 0.f), fmaxf(v[1], 0.f)), pack2(fmaxf(v[2], 0.f), fmaxf(v[3], 0.f)));
                continue;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int m = r0 + g + 8 * (q >> 1), o = c + (q & 1);
                if (m < n && o < out) Y[(size_t)m * out + o] = v[q];
            }
        }
        __syncthreads();
    }
}

// One tile of a layer per warp, between the flat FP32 parameters and the
// device's arrays: FP32 tiles and BF16 blocks from flat (pack), flat from the
// tiles (unpack).  blockIdx.y: layer, and those gridDim.y further on.
__device__ __forceinline__ void pack_layer(const MlpLayer& y, const float* flat, float4* w, float* bw) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, ot = y.doutp / 16, ki = y.dinp / 16;
    const int warps = gridDim.x * (blockDim.x / 32), w0 = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    for (int k = w0; k < ot * (y.dinp / 8); k += warps) {
        const int ob = k % ot, ib = k / ot;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int o = 16 * ob + g + 8 * (q >> 1), i = 8 * ib + 2 * t + (q & 1);
            v[q] = o < y.dout && i < y.din ? flat[y.woff + (long long)o * y.din + i] : 0.f;
        }
        w[(size_t)(y.tile + k) * 32 + lane] = make_float4(v[0], v[1], v[2], v[3]);
        __syncwarp();
        const uint32_t p0 = pack2(v[0], v[1]), p1 = pack2(v[2], v[3]);
        uint32_t* wp = reinterpret_cast<uint32_t*>(y.w + ((size_t)(2 * ob) * ki + ib / 2) * 32 + lane) + (ib & 1);
        wp[0] = p0;
        wp[(size_t)ki * 64] = p1;
        y.wt[((size_t)ib * ot + ob) * 32 + lane] = make_uint2(transpose8(p0), transpose8(p1));
    }
    for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < y.doutp; o += gridDim.x * blockDim.x)
        bw[y.bias + o] = o < y.dout ? flat[y.boff + o] : 0.f;
}

__global__ void pack_kernel(const MlpLayer* layers, int L, const float* flat, float4* w, float* bw) {
    for (int l = blockIdx.y; l < L; l += gridDim.y) pack_layer(layers[l], flat, w, bw);
}

__device__ __forceinline__ void unpack_layer(const MlpLayer& y, const float4* w, const float* bw, float* flat) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, ot = y.doutp / 16;
    const int warps = gridDim.x * (blockDim.x / 32), w0 = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    for (int k = w0; k < ot * (y.dinp / 8); k += warps) {
        const float4 f = w[(size_t)(y.tile + k) * 32 + lane];
        const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int o = 16 * (k % ot) + g + 8 * (q >> 1), i = 8 * (k / ot) + 2 * t + (q & 1);
            if (o < y.dout && i < y.din) flat[y.woff + (long long)o * y.din + i] = v[q];
        }
    }
    for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < y.dout; o += gridDim.x * blockDim.x)
        flat[y.boff + o] = bw[y.bias + o];
}
__global__ void unpack_kernel(const MlpLayer* layers, int L, const float4* w, const float* bw, float* flat) {
    for (int l = blockIdx.y; l < L; l += gridDim.y) unpack_layer(layers[l], w, bw, flat);
}

int pad16(int x) { return (x + 15) / 16 * 16; }

}  // namespace

struct bnm_mlp {
    int in = 0, hidden = 0, layers = 0, out = 0, max_batch = 0, device = 0;
    int L = 0;  // number of linear layers = layers + 1
    std::vector<MlpLayer> lay;
    MlpLayer* d_lay = nullptr;
    long long n_params = 0;
    int cluster = 8;        // CTAs of a cluster of mlp_step_kernel
    int fwd_clusters = 1;   // clusters of a forward pass: as many as the SMs would hold
    int width = 0;          // widest padded layer input
    size_t pred_smem = 0;   // shared memory of mlp_predict_kernel, 0: too wide for it
    size_t ahead_smem = 0;  // ... with the weights copied ahead, 0: too wide
    int ahead_rows = 0;     // ... for at most so many rows
    int pred_rows = 0;      // most rows per launch of mlp_predict_kernel
    int io_rows = 0;        // rows that io holds
    cudaStream_t st = nullptr;
    long long n_tiles = 0, n_bias = 0;
    float4 *w = nullptr, *m = nullptr, *v = nullptr;     // weights and Adam moments, [tile][lane]
    float *bw = nullptr, *bm = nullptr, *bv = nullptr;   // biases and theirs
    float* flat = nullptr;  // parameters or gradient in the caller's order: [W_l (out x in), b_l (out)]...
    float* yout = nullptr;  // [max_batch][out] last-layer output (f32)
    float* loss = nullptr;  // [kMaxSteps]
    float2* c12 = nullptr;  // [kMaxSteps]
    float *xin = nullptr, *tgt = nullptr;        // staged batch input / target (f32)
    float* tgt2 = nullptr;  // targets of the rows of two steps
    float *io = nullptr, *io_dev = nullptr;      // page-locked rows in and out of predict, as the device sees them
    float *data_x = nullptr, *data_y = nullptr;  // training set on the device
    long long data_n = 0;
    int* idx = nullptr;  // row indices of the steps of one launch
    size_t idx_cap = 0;
    int adam_t = 0;
    void* slab = nullptr;  // the device buffers above, except the growing ones (data_x, data_y, idx)
};

// Training steps per launch, and row indices of those steps (16 MB): bound the
// index buffer and the time one launch holds its SMs.
static constexpr int kMaxSteps = 2048;
static constexpr long long kMaxIdx = 4 << 20;

static void free_io(bnm_mlp* p) {
    if (p->io) {
        cudaHostUnregister(p->io);
        std::free(p->io);
    }
    p->io = p->io_dev = nullptr;
    p->io_rows = 0;
}

extern "C" void bnm_mlp_destroy(bnm_mlp* p) {
    if (!p) return;
    cudaSetDevice(p->device);
    if (p->st) cudaStreamSynchronize(p->st);
    for (void* a : {p->slab, (void*)p->data_x, (void*)p->data_y, (void*)p->idx})
        if (a) cudaFree(a);
    free_io(p);
    if (p->st) cudaStreamDestroy(p->st);
    delete p;
}

static dim3 layer_grid(const bnm_mlp* p) { return dim3(64, (unsigned)std::min(p->L, 65535)); }  // the grid's limit

// Device arrays from the flat parameters, Adam's state cleared (asynchronous)
static cudaError_t load_flat(bnm_mlp* p) {
    pack_kernel<<<layer_grid(p), 256, 0, p->st>>>(p->d_lay, p->L, p->flat, p->w, p->bw);
    cudaError_t e = cudaGetLastError();
    // m, v, bm, bv follow one another in the slab
    if (e == cudaSuccess)
        e = cudaMemsetAsync(p->m, 0, (size_t)((char*)(p->bv + p->n_bias) - (char*)p->m), p->st);
    return e;
}

static int mlp_init(bnm_mlp* p, uint64_t seed) {
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    BNM_CUDA_TRY(cudaStreamCreateWithFlags(&p->st, cudaStreamNonBlocking));
    const size_t np = (size_t)p->n_params, rows = pad16(p->max_batch);
    const size_t tb = (size_t)p->n_tiles * 32 * sizeof(float4), bb = (size_t)p->n_bias * 4;
    // every buffer is a piece of one allocation: sized first, then placed
    for (int pass = 0; pass < 2; pass++) {
        unsigned char* base = pass ? static_cast<unsigned char*>(p->slab) : nullptr;
        size_t off = 0;
        auto take = [&](auto*& field, size_t bytes) {
            if (pass) field = reinterpret_cast<std::remove_reference_t<decltype(field)>>(base + off);
            off += (bytes + 255) / 256 * 256;
        };
        take(p->m, tb);
        take(p->v, tb);
        take(p->bm, bb);
        take(p->bv, bb);
        take(p->w, tb);
        take(p->bw, bb);
        take(p->flat, np * 4);
        for (MlpLayer& y : p->lay) {
            take(y.w, (size_t)y.dinp * y.doutp * 2);
            take(y.wt, (size_t)y.dinp * y.doutp * 2);
            p->width = std::max(p->width, y.dinp);
        }
        take(p->yout, (size_t)p->max_batch * p->out * 4);
        take(p->loss, (size_t)kMaxSteps * 4);
        take(p->c12, (size_t)kMaxSteps * 8);
        take(p->xin, (size_t)p->max_batch * p->in * 4);
        take(p->tgt, (size_t)p->max_batch * p->out * 4);
        take(p->tgt2, (size_t)2 * p->max_batch * p->out * 4);
        for (MlpLayer& y : p->lay) {
            const size_t sets = &y == &p->lay[0] ? 2 : 1;
            take(y.x, sets * rows * y.dinp * 2);
            take(y.xt, sets * rows * y.dinp * 2);
            take(y.dz, (size_t)p->max_batch * y.doutp * 4);
            take(y.dzh, rows * y.doutp * 2);
            take(y.dzt, rows * y.doutp * 2);
        }
        take(p->d_lay, p->lay.size() * sizeof(MlpLayer));
        if (!pass) BNM_CUDA_TRY(cudaMalloc(&p->slab, off));
    }
    BNM_CUDA_TRY(cudaMemcpyAsync(p->d_lay, p->lay.data(), p->lay.size() * sizeof(MlpLayer), cudaMemcpyHostToDevice,
                                 p->st));
    // predict: rows travel through a page-locked buffer of at most 1 MiB, made
    // by what the calls ask for, because locking is paid by an object's first
    // call: registered memory, 512 rows of 19 inputs, 0.55 ms; cudaMallocHost for
    // the largest call an object might make, 2.7 ms (any size up to 2 MB takes
    // it 1.2-2.9 ms; 16 MiB 7-20).
    const size_t row_bytes = (size_t)(p->in + p->out) * 4;
    p->pred_rows = (int)std::max<size_t>(16, ((size_t)1 << 20) / row_bytes / 16 * 16);
    int sms = 0;
    BNM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device));
    p->pred_smem = (size_t)2 * 16 * p->width * 2;
    if (p->pred_smem > 200 * 1024) p->pred_smem = 0;
    if (p->pred_smem) {
        BNM_CUDA_TRY(cudaFuncSetAttribute(mlp_predict_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          200 * 1024));
        const size_t ahead = p->pred_smem + (size_t)kPredWarps * kPredDepth * p->width * 2 * sizeof(uint2);
        if (ahead <= 210 * 1024) {
            BNM_CUDA_TRY(cudaFuncSetAttribute(mlp_predict_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              210 * 1024));
            p->ahead_smem = ahead;
            p->ahead_rows = 16 * sms;
        }
    }
    // 16 CTAs where the GPU can place such a cluster, else the portable 8
    BNM_CUDA_TRY(cudaFuncSetAttribute(mlp_step_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kStepThreads);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, mlp_step_kernel, &cfg) == cudaSuccess && clusters > 0)
        p->cluster = 16;
    cudaGetLastError();
    p->fwd_clusters = std::max(1, sms / p->cluster);
    // He-uniform initialisation (host, seeded), zero biases; Adam state zero
    std::vector<float> w0(np, 0.f);
    std::mt19937_64 gen(seed);
    for (const MlpLayer& y : p->lay) {
        const float lim = std::sqrt(6.0f / (float)y.din);
        std::uniform_real_distribution<float> U(-lim, lim);
        for (long long i = 0; i < (long long)y.din * y.dout; i++) w0[y.woff + i] = U(gen);
    }
    BNM_CUDA_TRY(cudaMemcpyAsync(p->flat, w0.data(), np * 4, cudaMemcpyHostToDevice, p->st));
    BNM_CUDA_TRY(load_flat(p));
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    return BNM_OK;
}

extern "C" int bnm_mlp_create(int32_t in_dim, int32_t hidden, int32_t layers, int32_t out_dim, int32_t max_batch,
                              uint64_t seed, int32_t device, bnm_mlp** out) {
    if (!out || in_dim < 1 || hidden < 1 || layers < 1 || out_dim < 1 || max_batch < 1)
        return bnm_fail_msg(BNM_EINVAL, "bad MLP sizes");
    *out = nullptr;
    bnm_mlp* p = new bnm_mlp();
    p->in = in_dim;
    p->hidden = hidden;
    p->layers = layers;
    p->out = out_dim;
    p->max_batch = max_batch;
    p->device = device;
    p->L = layers + 1;
    for (int l = 0; l < p->L; l++) {
        MlpLayer y;
        std::memset(&y, 0, sizeof y);
        y.din = l == 0 ? in_dim : hidden;
        y.dout = l == p->L - 1 ? out_dim : hidden;
        y.dinp = pad16(y.din);
        y.doutp = pad16(y.dout);
        y.woff = p->n_params;
        p->n_params += (long long)y.din * y.dout;
        y.boff = p->n_params;
        p->n_params += y.dout;
        y.tile = p->n_tiles;
        p->n_tiles += (long long)(y.doutp / 16) * (y.dinp / 8);
        y.bias = p->n_bias;
        p->n_bias += y.doutp;
        p->lay.push_back(y);
    }
    const int rc = mlp_init(p, seed);
    if (rc) {
        bnm_mlp_destroy(p);
        return rc;
    }
    *out = p;
    return BNM_OK;
}

static StepArgs step_args(bnm_mlp* p, int mode, int batch, const float* X, const float* T) {
    StepArgs a;
    std::memset(&a, 0, sizeof a);
    a.layers = p->d_lay;
    a.L = p->L;
    a.in = p->in;
    a.out = p->out;
    a.mode = mode;
    a.steps = 1;
    a.batch = batch;
    a.w = p->w;
    a.m = p->m;
    a.v = p->v;
    a.bw = p->bw;
    a.bm = p->bm;
    a.bv = p->bv;
    a.g = p->flat;
    a.X = X;
    a.T = T;
    a.c12 = p->c12;
    a.x0 = (size_t)pad16(p->max_batch) * p->lay[0].dinp * 2 / sizeof(uint4);
    a.xt0 = 2 * a.x0;
    a.tgt = p->tgt2;
    a.yout = p->yout;
    a.loss = p->loss;
    return a;
}

static int launch_step(bnm_mlp* p, const StepArgs& a, int clusters = 1) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p->cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(p->cluster * clusters));
    cfg.blockDim = dim3(kStepThreads);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = p->st;
    BNM_CUDA_TRY(cudaLaunchKernelEx(&cfg, mlp_step_kernel, a));
    return BNM_OK;
}

// Makes io hold at least `rows` rows (no fewer than 64 KB, or twice what it held);
// false: no page-locked memory to be had, rows go through pageable copies.
static bool pred_buffer(bnm_mlp* p, int rows) {
    if (p->io_rows >= rows) return true;
    const size_t row_bytes = (size_t)(p->in + p->out) * 4;
    rows = std::min(p->pred_rows, std::max(rows, std::max(2 * p->io_rows, (int)((64 << 10) / row_bytes))));
    free_io(p);
    void *h = std::aligned_alloc(4096, (rows * row_bytes + 4095) / 4096 * 4096), *d = nullptr;
    if (!h) return false;
    cudaError_t e = cudaHostRegister(h, rows * row_bytes, cudaHostRegisterMapped);
    if (e == cudaSuccess && (e = cudaHostGetDevicePointer(&d, h, 0)) != cudaSuccess) cudaHostUnregister(h);
    if (e != cudaSuccess) {
        cudaGetLastError();
        std::free(h);
        return false;
    }
    p->io = static_cast<float*>(h);
    p->io_dev = static_cast<float*>(d);
    p->io_rows = rows;
    return true;
}

extern "C" int bnm_mlp_predict(bnm_mlp* p, const float* X, int32_t n, float* Y) {
    if (!p || !X || !Y || n < 0) return bnm_fail_msg(BNM_EINVAL, "bad predict arguments");
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    // rows in a launch of the forward kernel, 0: too wide for it
    auto forward = [&](const float* x, float* y, int B) -> cudaError_t {
        // Copying ahead takes most of an SM's shared memory, so it is for
        // calls of at most one CTA per SM; beyond, several CTAs per SM hide
        // the loads of one another (8192 rows: 120 us with, 98 us without; 2368: 53 and 52).
        const bool ahead = B <= p->ahead_rows;
        (ahead ? mlp_predict_kernel<true> : mlp_predict_kernel<false>)<<<
            (B + 15) / 16, kPredThreads, ahead ? p->ahead_smem : p->pred_smem, p->st>>>(p->d_lay, p->L, p->in, p->out,
                                                                                      B, p->width, p->bw, x, y);
        return cudaGetLastError();
    };
    // Rows through locked memory, read and written there by the kernel (512 rows:
    // 0.04 ms), or, for calls that exceed the locked buffer where the device's holds
    // more, through that and pageable copies (8192 rows of 1000 inputs: 1.7 ms, 3.3
    // locked in pieces; 65,536 of 19 0.59 and 0.86).
    const bool locked = p->pred_smem && (n <= p->pred_rows || p->max_batch < p->pred_rows);
    if (locked && pred_buffer(p, std::min(n, p->pred_rows))) {
        const int rows = p->io_rows;
        const size_t y = (size_t)rows * p->in;  // the outputs follow the inputs
        for (int s = 0; s < n; s += rows) {
            const int B = std::min(rows, n - s);
            std::memcpy(p->io, X + (size_t)s * p->in, (size_t)B * p->in * 4);
            BNM_CUDA_TRY(forward(p->io_dev, p->io_dev + y, B));
            BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
            std::memcpy(Y + (size_t)s * p->out, p->io + y, (size_t)B * p->out * 4);
        }
        return BNM_OK;
    }
    for (int s = 0; s < n; s += p->max_batch) {
        const int B = std::min(p->max_batch, n - s);
        BNM_CUDA_TRY(cudaMemcpyAsync(p->xin, X + (size_t)s * p->in, (size_t)B * p->in * 4, cudaMemcpyHostToDevice, p->st));
        if (p->pred_smem) {
            BNM_CUDA_TRY(forward(p->xin, p->yout, B));
        } else {
            int rc = launch_step(p, step_args(p, kForward, B, p->xin, nullptr), std::min(p->fwd_clusters, (B + 31) / 32));
            if (rc) return rc;
        }
        BNM_CUDA_TRY(cudaMemcpyAsync(Y + (size_t)s * p->out, p->yout, (size_t)B * p->out * 4, cudaMemcpyDeviceToHost, p->st));
    }
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    return BNM_OK;
}

extern "C" int bnm_mlp_loss_and_grads(bnm_mlp* p, const float* X, const float* T, int32_t n, float* loss,
                                      float* grads) {
    if (!p || !X || !T || n < 1 || n > p->max_batch) return bnm_fail_msg(BNM_EINVAL, "batch must be in [1, max_batch]");
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    BNM_CUDA_TRY(cudaMemcpyAsync(p->xin, X, (size_t)n * p->in * 4, cudaMemcpyHostToDevice, p->st));
    BNM_CUDA_TRY(cudaMemcpyAsync(p->tgt, T, (size_t)n * p->out * 4, cudaMemcpyHostToDevice, p->st));
    int rc = launch_step(p, step_args(p, kGrads, n, p->xin, p->tgt));
    if (rc) return rc;
    if (loss) BNM_CUDA_TRY(cudaMemcpyAsync(loss, p->loss, 4, cudaMemcpyDeviceToHost, p->st));
    if (grads) BNM_CUDA_TRY(cudaMemcpyAsync(grads, p->flat, (size_t)p->n_params * 4, cudaMemcpyDeviceToHost, p->st));
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    return BNM_OK;
}

extern "C" int bnm_mlp_train(bnm_mlp* p, const float* X, const float* Y, int32_t n, int32_t epochs, int32_t batch,
                             float lr, uint64_t shuffle_seed, float* loss_per_epoch) {
    if (!p || !X || !Y || n < 1 || batch < 1 || batch > p->max_batch || epochs < 0)
        return bnm_fail_msg(BNM_EINVAL, "bad training arguments");
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    const int nb = n / batch;  // full batches only
    if (p->data_n < n) {
        for (float** q : {&p->data_x, &p->data_y}) {
            if (*q) cudaFree(*q);
            *q = nullptr;
        }
        p->data_n = 0;
        BNM_CUDA_TRY(cudaMalloc(&p->data_x, (size_t)n * p->in * 4));
        BNM_CUDA_TRY(cudaMalloc(&p->data_y, (size_t)n * p->out * 4));
        p->data_n = n;
    }
    const long long total = (long long)nb * epochs;
    const int max_steps = (int)std::max<long long>(1, std::min<long long>(kMaxSteps, kMaxIdx / batch));
    const size_t need = (size_t)std::min<long long>(total, max_steps) * batch;
    if (p->idx_cap < need) {
        if (p->idx) cudaFree(p->idx);
        p->idx = nullptr;
        p->idx_cap = 0;
        BNM_CUDA_TRY(cudaMalloc(&p->idx, need * 4));
        p->idx_cap = need;
    }
    BNM_CUDA_TRY(cudaMemcpyAsync(p->data_x, X, (size_t)n * p->in * 4, cudaMemcpyHostToDevice, p->st));
    BNM_CUDA_TRY(cudaMemcpyAsync(p->data_y, Y, (size_t)n * p->out * 4, cudaMemcpyHostToDevice, p->st));
    std::vector<int> order(n), idx;
    for (int i = 0; i < n; i++) order[i] = i;
    std::mt19937_64 gen(shuffle_seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    std::vector<float2> c12;
    std::vector<float> losses((size_t)total);
    long long done = 0;
    // one launch per max_steps steps
    auto flush = [&]() -> int {
        const int steps = (int)c12.size();
        if (!steps) return BNM_OK;
        BNM_CUDA_TRY(cudaMemcpyAsync(p->idx, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice, p->st));
        BNM_CUDA_TRY(cudaMemcpyAsync(p->c12, c12.data(), (size_t)steps * 8, cudaMemcpyHostToDevice, p->st));
        StepArgs a = step_args(p, kTrain, batch, p->data_x, p->data_y);
        a.steps = steps;
        a.idx = p->idx;
        a.lr = lr;
        a.b1 = b1;
        a.b2 = b2;
        a.eps = eps;
        int rc = launch_step(p, a);
        if (rc) return rc;
        BNM_CUDA_TRY(cudaMemcpyAsync(losses.data() + done, p->loss, (size_t)steps * 4, cudaMemcpyDeviceToHost, p->st));
        BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
        done += steps;
        idx.clear();
        c12.clear();
        return BNM_OK;
    };
    int rc;
    for (int ep = 0; ep < epochs; ep++) {
        std::shuffle(order.begin(), order.end(), gen);
        for (int s = 0; s < nb; s++) {
            idx.insert(idx.end(), order.begin() + (size_t)s * batch, order.begin() + (size_t)(s + 1) * batch);
            p->adam_t++;
            c12.push_back(make_float2(1.f - std::pow(b1, (float)p->adam_t), 1.f - std::pow(b2, (float)p->adam_t)));
            if ((int)c12.size() == max_steps && (rc = flush())) return rc;
        }
    }
    if ((rc = flush())) return rc;
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    for (int ep = 0; loss_per_epoch && ep < epochs; ep++) {
        double sum = 0.0;
        for (int s = 0; s < nb; s++) sum += losses[(size_t)ep * nb + s];
        loss_per_epoch[ep] = nb ? (float)(sum / nb) : 0.f;
    }
    return BNM_OK;
}

extern "C" int64_t bnm_mlp_num_params(const bnm_mlp* p) { return p ? p->n_params : 0; }

extern "C" int bnm_mlp_get_params(bnm_mlp* p, float* flat) {
    if (!p || !flat) return bnm_fail_msg(BNM_EINVAL, "null argument");
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    unpack_kernel<<<layer_grid(p), 256, 0, p->st>>>(p->d_lay, p->L, p->w, p->bw, p->flat);
    BNM_CUDA_TRY(cudaGetLastError());
    BNM_CUDA_TRY(cudaMemcpyAsync(flat, p->flat, (size_t)p->n_params * 4, cudaMemcpyDeviceToHost, p->st));
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    return BNM_OK;
}

extern "C" int bnm_mlp_set_params(bnm_mlp* p, const float* flat) {
    if (!p || !flat) return bnm_fail_msg(BNM_EINVAL, "null argument");
    BNM_CUDA_TRY(cudaSetDevice(p->device));
    BNM_CUDA_TRY(cudaMemcpyAsync(p->flat, flat, (size_t)p->n_params * 4, cudaMemcpyHostToDevice, p->st));
    // new parameters start a new optimisation: Adam's moments and step count restart
    p->adam_t = 0;
    BNM_CUDA_TRY(load_flat(p));
    BNM_CUDA_TRY(cudaStreamSynchronize(p->st));
    return BNM_OK;
}
