// Reference-order integrator (any N up to 1024, float or double).
//
// One CTA integrates one particle at a time (persistent: CTAs pull particle
// indices from a global counter).  It restates the
// reference's time loop (bnm.cpp:167-290; the same model as bnm.cu:72-315)
// with the reference's operand order and operand types, and it is compiled
// with -fmad=false in integrate_exact.cu, so that in double it reproduces the
// reference's FP64 CPU arithmetic up to the last-ulp differences of the
// device exp/pow, and in float the reference's USE_FLOATS arithmetic.  It is
// the parity path (oracle-noise mode, step-for-step checks) and the fallback
// for node counts the register-resident fast kernel does not cover.
//
// Semantics that follow the reference's CPU path rather than its GPU path
// (bnm.cu differs in these places):
//   * numerical FIC: delta is rounded through fmaxf (bnm.cpp:250) and the
//     per-node extended sums restart with the simulation after an FIC trial
//     (the CPU keeps only the final time series, bnm.cpp:212-226);
//   * no FP32 clamp of |aI-b| < 1e-4 (bnm.cu:195-199 only).
//
// What bounds it: a substep is a chain, the N products of a node's coupling
// added one after the other in the reference's order, then exp, a division and
// the state update, in FP64 with no contraction.  With one thread per node,
// both populations in it and the SC rows in shared memory as they come, a
// substep took 3.0 us at N = 100 (FP64, 8 particles): the lanes' row reads
// conflict (stride N doubles), the noise was loaded where it was used, and the
// inhibitory exp and division and the Balloon-Windkessel powers stood in the
// same thread's way.  Now (kSplit) warps of their own hold the inhibitory
// population and the BOLD state, which need the excitatory gating only from
// the substep before; SC is kept transposed (kSmem), so a warp's reads are
// consecutive; noise is loaded a substep ahead; and every term that does not
// need the coupling is formed before it.  The operations and their order per
// value are unchanged.  N = 100, FP64, 8 particles of 8 s: 254 -> 106 ms (1.31 us
// a substep; the products alone are a chain of 100 additions of 9 cycles).
#pragma once
#include "bnm_common.cuh"

// Each translation unit that includes this header instantiates its own copy
// (integrate_exact.cu with -fmad=false, integrate_fast.cu with contraction),
// so the kernels live in a per-TU namespace.
#ifndef BNM_GENERIC_NS
#error "define BNM_GENERIC_NS before including integrate_generic.cuh"
#endif

namespace bnm {
namespace BNM_GENERIC_NS {

__device__ __forceinline__ float dexp(float x) { return expf(x); }
__device__ __forceinline__ double dexp(double x) { return exp(x); }
__device__ __forceinline__ float dpow(float a, float b) { return powf(a, b); }
__device__ __forceinline__ double dpow(double a, double b) { return pow(a, b); }

template <typename R>
__device__ __forceinline__ const R* sc_ptr(const SimArgs& a);
template <>
__device__ __forceinline__ const float* sc_ptr<float>(const SimArgs& a) { return a.sc_f32; }
template <>
__device__ __forceinline__ const double* sc_ptr<double>(const SimArgs& a) { return a.sc_f64; }

template <typename R>
__device__ __forceinline__ void store_bold(const SimArgs& a, size_t idx, R v);
template <>
__device__ __forceinline__ void store_bold<float>(const SimArgs& a, size_t idx, float v) { a.bold[idx] = v; }
template <>
__device__ __forceinline__ void store_bold<double>(const SimArgs& a, size_t idx, double v) { a.bold_f64[idx] = v; }

// Coupling of one node, the products added in column order, SC in global
// memory, its columns `step` values apart.
template <typename R>
__device__ __forceinline__ R dot_global(const R* sc, int step, const R* S, int N) {
    R c = 0;
#pragma unroll 8
    for (int k = 0; k < N; k++) c += sc[(size_t)k * step] * S[k];
    return c;
}

// 16 bytes of consecutive columns.
template <typename R>
struct __align__(16) Vec {
    static constexpr int n = 16 / sizeof(R);
    R x[n];
};
constexpr int kColPad = 4;  // columns in shared memory, rounded up (zero SC and S)

// The same from shared memory, SC as Vecs [column / n][node]: a warp's reads
// are consecutive, S is broadcast.  Groups of 32 bytes (8 FP32 or 4 FP64
// columns) are loaded two ahead of the chain of additions.  The padding adds
// +0 to the sum, which changes no bit of it (it starts at +0).
template <typename R>
__device__ __forceinline__ R dot_smem(const Vec<R>* sc, int nodes, const R* S, int cols) {
    constexpr int V = Vec<R>::n, U = kColPad * (int)sizeof(R) / 16;  // Vecs of one group of kColPad columns
    const Vec<R>* s = reinterpret_cast<const Vec<R>*>(S);
    struct Group {
        Vec<R> v[U], s[U];
    };
    auto load = [&](Group& g) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            g.v[u] = *sc;
            g.s[u] = *s++;
            sc += nodes;
        }
    };
    R c = 0;
    auto add = [&](const Group& g) {
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int k = 0; k < V; k++) c += g.v[u].x[k] * g.s[u].x[k];
    };
    Group g0, g1, g2;
    const int n = cols / kColPad;
    load(g0);
    if (n > 1) load(g1);
    int k = 0;
    for (; k + 5 <= n; k += 3) {  // groups k, k + 1 are loaded
        load(g2);
        add(g0);
        load(g0);
        add(g1);
        load(g1);
        add(g2);
    }
    // up to four groups are left, two of them loaded
    const int left = n - k;
    if (left > 2) load(g2);
    add(g0);
    if (left > 3) load(g0);
    if (left > 1) add(g1);
    if (left > 2) add(g2);
    if (left > 3) add(g0);
    return c;
}

// Dynamic shared memory: S_E[2][npad], S_I[2][npad] (+ SC[cols / n][N] Vecs when
// kSmem).  kSplit: two threads a node, kThreads the largest CTA.
template <typename R, bool kSplit, bool kSmem, int kThreads>
__global__ void __launch_bounds__(kThreads) integrate_generic_kernel(SimArgs a) {
    typedef Model<R> C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int N = a.N, npad = kSplit ? blockDim.x / 2 : blockDim.x;
    // SC in global memory: FP32 by rows (shared with the other integrators), FP64 by columns
    const int row = sizeof(R) == 4 ? a.sc_ld : 1, step = sizeof(R) == 4 ? 1 : N;
    R* S_buf = reinterpret_cast<R*>(smem_raw);
    R* I_buf = S_buf + 2 * npad;
    const R* SC = sc_ptr<R>(a);
    const int cols = (N + kColPad - 1) / kColPad * kColPad;
    if (kSmem) {
        constexpr int V = Vec<R>::n;
        R* sc_s = I_buf + 2 * npad;
        for (int i = threadIdx.x; i < N * cols; i += blockDim.x) {
            // consecutive threads take what is consecutive in global memory
            const int r = sizeof(R) == 4 ? i / cols : i % N, c = sizeof(R) == 4 ? i % cols : i / N;
            sc_s[((c / V) * N + r) * V + c % V] = c < N ? SC[(size_t)r * row + (size_t)c * step] : (R)0;
        }
        SC = sc_s;
    }
    __shared__ int s_sim;
    // excitatory role: coupling, S_E, FIC; inhibitory role: S_I, BOLD
    const bool isE = !kSplit || (int)threadIdx.x < npad, isI = !kSplit || !isE;
    const int j = kSplit && !isE ? threadIdx.x - npad : threadIdx.x;
    const bool act = j < N;
    const R* sc_row = SC + (size_t)(act ? j : 0) * (kSmem ? Vec<R>::n : row);
    const unsigned int duration = a.samp_end - a.samp_start + 1;
    const size_t plane = (size_t)a.noise_ld;  // node stride of the noise table
    // noise of this thread's node: both values, or its own population's
    const float* nz_base = a.noise + 2 * j + (kSplit && !isE ? 1 : 0);
    const long long n_sub = ((long long)a.T + 1) * 10;

    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_sim = atomicAdd(a.work_counter, 1);
        __syncthreads();
        const int sim = s_sim;
        if (sim >= a.n_sims) break;

        const R G = (R)a.G[sim];
        const R wEE = act ? (R)a.wEE[(size_t)sim * N + j] : (R)0;
        const R wEI = act ? (R)a.wEI[(size_t)sim * N + j] : (R)0;
        R wIE = act ? (R)a.wIE[(size_t)sim * N + j] : (R)0;
        R S_E = 0.001, S_I = 0.001, x = 0.0, f = 1.0, nu = 1.0, q = 1.0;
        R IE = 0, II = 0, rE = 0, rI = 0, mean_IE = 0, delta = (R)a.init_delta;
        R ext[6] = {0, 0, 0, 0, 0, 0};
        if (isE) {
            S_buf[j] = act ? S_E : (R)0;
            S_buf[npad + j] = (R)0;
        }
        if (kSplit && isI) I_buf[j] = I_buf[npad + j] = S_I;
        int cur = 0, trial = 0, ts = 0, frame = 0;
        bool failed = false, adjusting = a.adjust_fic != 0;
        // noise of the coming substep
        float n0 = 0.f, n1 = 0.f;
        auto fetch = [&](long long sub) {
            if (!act || sub >= n_sub) return;
            const float* p = nz_base + (size_t)sub * plane * 2;
            n0 = p[0];
            if (!kSplit) n1 = p[1];
        };
        fetch(0);
        __syncthreads();

        while (ts <= a.T) {
            for (int sub = 0; sub < 10; sub++) {
                if (act) {
                    const R* Sp = S_buf + cur * npad;
                    if (kSplit && isE) S_I = I_buf[cur * npad + j];
                    if (kSplit && isI) S_E = Sp[j];
                    const R nE = (R)n0, nI = (R)(kSplit ? n0 : n1);
                    fetch((long long)ts * 10 + sub + 1);
                    // terms without the coupling, then the inhibitory population
                    R base = 0, inh = 0, zE = 0, leakE = 0, inE = 0, newI = 0;
                    if (isE) {
                        base = C::w_E__I_0 + wEE * S_E;
                        inh = wIE * S_I;
                        zE = nE * C::sigma_model * C::sqrt_dt;
                        leakE = S_E / C::tau_E;
                        inE = (1 - S_E) * C::gamma_E;
                    }
                    if (isI) {
                        II = C::w_I__I_0 + wEI * S_E - S_I;
                        R eI = dexp(-C::d_I * (C::a_I * II - C::b_I));
                        rI = (C::a_I * II - C::b_I) / (1 - eI);
                        R dSI = nI * C::sigma_model * C::sqrt_dt + C::dt * (C::gamma_I * rI - (S_I / C::tau_I));
                        newI = S_I + dSI;
                        // std::max(0, std::min(S, 1)) of bnm.cpp:195-199, NaN -> 0 included
                        newI = ((R)1.0 < newI) ? (R)1.0 : newI;
                        newI = ((R)0.0 < newI) ? newI : (R)0.0;
                    }
                    if (isE) {
                        R coupling;
                        if constexpr (kSmem)
                            coupling = dot_smem<R>(reinterpret_cast<const Vec<R>*>(sc_row), N, Sp, cols);
                        else
                            coupling = dot_global<R>(sc_row, step, Sp, N);
                        IE = base + coupling * G * C::J_NMDA - inh;
                        R eE = dexp(-C::d_E * (C::a_E * IE - C::b_E));
                        rE = (C::a_E * IE - C::b_E) / (1 - eE);
                        R dSE = zE + C::dt * (inE * rE - leakE);
                        S_E += dSE;
                        S_E = ((R)1.0 < S_E) ? (R)1.0 : S_E;
                        S_E = ((R)0.0 < S_E) ? S_E : (R)0.0;
                        S_buf[(cur ^ 1) * npad + j] = S_E;
                    }
                    if (isI) {
                        S_I = newI;
                        if (kSplit) I_buf[(cur ^ 1) * npad + j] = S_I;
                    }
                }
                __syncthreads();
                cur ^= 1;
            }
            // the inhibitory role's copy of S_E for the BOLD state
            if (kSplit && isI && act) S_E = S_buf[cur * npad + j];
            if (act && isI) {
                // Balloon-Windkessel once per ms (bnm.cpp:204-211); the double
                // literals promote exactly as in the reference.
                x = x + C::model_dt * (S_E - C::kappa * x - C::y * (f - 1.0));
                R tmp_f = f + C::model_dt * x;
                nu = nu + C::model_dt * C::itau * (f - dpow(nu, C::ialpha));
                q = q + C::model_dt * C::itau *
                            (f * (1.0 - dpow(C::oneminrho, (R)(1.0 / f))) / C::rho - dpow(nu, C::ialpha) * q / nu);
                f = tmp_f;
            }
            if (ts % a.TR == 0) {
                if (act && isI) {
                    R b = C::V_0 * (C::k1 * (1 - q) + C::k2 * (1 - q / nu) + C::k3 * (1 - nu));
                    store_bold<R>(a, ((size_t)sim * a.frames + frame) * N + j, b);
                }
                if (act && frame >= a.n_vols_remove) {  // a role's own three are written out
                    ext[0] += S_E;
                    ext[1] += IE;
                    ext[2] += rE;
                    ext[3] += S_I;
                    ext[4] += II;
                    ext[5] += rI;
                }
                frame++;
            }
            ts++;
            if (adjusting) {
                if (ts >= a.samp_start && ts <= a.samp_end) mean_IE += IE;
                if (ts == a.samp_end) {
                    bool needs = false;
                    if (act && isE) {
                        mean_IE /= duration;
                        R diff = mean_IE - C::b_a_ratio_E;
                        if (fabs(diff + 0.026) > 0.005) {
                            needs = true;
                            if (trial < a.max_trials) {
                                if (diff < -0.026) {
                                    wIE -= delta;
                                    delta -= 0.001;
                                    delta = fmaxf(delta, 0.001);
                                } else {
                                    wIE += delta;
                                }
                            }
                        }
                    }
                    if (__syncthreads_or(needs)) {
                        if (trial < a.max_trials) {
                            S_E = 0.001;
                            S_I = 0.001;
                            x = 0.0;
                            f = 1.0;
                            nu = 1.0;
                            q = 1.0;
                            mean_IE = 0;
                            for (int v = 0; v < 6; v++) ext[v] = 0;
                            if (act && isE) S_buf[cur * npad + j] = S_E;
                            if (act && kSplit && isI) I_buf[cur * npad + j] = S_I;
                            fetch(0);
                            ts = 0;
                            frame = 0;
                            trial++;
                        } else {
                            failed = true;
                            adjusting = false;
                        }
                    } else {
                        adjusting = false;
                    }
                    __syncthreads();
                }
            }
        }
        if (act) {
            if (isE) a.wIE_out[(size_t)sim * N + j] = (double)wIE;
            const int kept = frame - a.n_vols_remove;
#pragma unroll
            for (int v = 0; v < 6; v++) {
                if (v < 3 ? !isE : !isI) continue;
                R m = ext[v];
                m /= kept;
                a.ext[((size_t)sim * 6 + v) * N + j] = (double)m;
            }
        }
        if (threadIdx.x == 0) {
            a.trials[sim] = trial;
            a.failed[sim] = failed ? 1 : 0;
        }
    }
}

template <typename R, bool kSplit, bool kSmem, int kThreads>
static cudaError_t launch_generic_t(const SimArgs& a, int threads, size_t smem, int num_sms, cudaStream_t st) {
    auto* fn = integrate_generic_kernel<R, kSplit, kSmem, kThreads>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = a.n_sims < 2 * num_sms ? a.n_sims : 2 * num_sms;
    fn<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}
// The variant for N nodes and n particles:
//   SC in shared memory where it fits an SM (FP64 up to 164 nodes, FP32 up to
//   234), two threads a node;
//   else SC from global memory, two threads a node up to 256 nodes.  In FP64
//   that takes 122 registers a thread and an SM holds one CTA, where it held
//   two with one thread a node; with SC by rows, a cache line per lane, that
//   cost calls of more particles than SMs (N = 200, 296 particles of 600 ms: 176
//   ms with one thread a node, 193 with two).  By columns the L1 no longer
//   bounds it: 81 ms, and 40 with 148 particles (103 and 96 by rows);
//   else one thread a node: FP64 with 96 registers while the CTA leaves each
//   thread that many (640 threads), above with 64 and some spills.
template <typename R>
static cudaError_t launch_generic(const SimArgs& a, int num_sms, cudaStream_t st) {
    const int npad = ((a.N + 31) / 32) * 32;
    if (npad > 1024) return cudaErrorInvalidValue;
    const size_t smem = 4 * (size_t)npad * sizeof(R);
    const size_t sc_bytes = (size_t)a.N * ((a.N + kColPad - 1) / kColPad * kColPad) * sizeof(R);
    if (smem + sc_bytes <= 220 * 1024)
        return launch_generic_t<R, true, true, 512>(a, 2 * npad, smem + sc_bytes, num_sms, st);
    if (npad <= 256) return launch_generic_t<R, true, false, 512>(a, 2 * npad, smem, num_sms, st);
    if constexpr (sizeof(R) == 8)
        if (npad <= 640) return launch_generic_t<R, false, false, 640>(a, npad, smem, num_sms, st);
    return launch_generic_t<R, false, false, 1024>(a, npad, smem, num_sms, st);
}

}  // namespace BNM_GENERIC_NS
}  // namespace bnm
