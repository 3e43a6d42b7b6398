// Differentiable N-turn map and its hand-written adjoint.
//
// One turn t of the forward map, in the reference main loop's order
// (blond/impedances/impedance.py:113-146 then blond/trackers/tracker.py:
// 521-615: induced voltage of the turn-start profile, linear_interp_kick,
// RF kick, drift):
//
//   p_t      = CIC(dt_t)                          profile (counts)
//   V_t      = -s irfft(Z rfft(p_t, n_fft))[:S]   induced voltage, s = q e ratio
//   dE'      = dE_t + q interp(V_t; dt_t) + q sum_j V_j sin(w_j dt_t + phi_j) + acc_t
//   dt_t+1   = dt_t + c_t dE',  dE_t+1 = dE'       simple drift, c_t from turn t+1
//
// CIC is cloud-in-cell deposition on the profile's bin centres
// bc_k = bc_0 + k w: a particle at f = (dt - bc_0)/w gives 1 - u to bin
// floor(f) and u = f - floor(f) to the next, so the profile is continuous
// and piecewise linear in every dt.  (The reference's smooth_histogram,
// blond/cpp_routines/histogram.cpp:75-132, moves a whole particle by two
// bins where it crosses a bin centre, so its profile has no useful
// derivative.)  interp(V; dt) = V_k (1 - u) + V_k+1 u on the same grid is
// the function of linear_interp_kick.cpp:44-62, written without the
// slope/offset cancellation.
//
// The adjoint of one turn, lambda = dL/d(state), runs backwards:
//
//   lambda_dt    += (lambda_p_t+1[k+1] - lambda_p_t+1[k]) / w   at dt_t+1
//   lambda_dE'    = lambda_dE + c_t lambda_dt
//   lambda_dt    += lambda_dE' q (sum_j V_j w_j cos(.) + (V_k+1 - V_k) / w)
//   dL/dV_j,t    += sum_i lambda_dE' q sin(.)
//   dL/dphi_j,t  += sum_i lambda_dE' q V_j cos(.)
//   lambda_V[k]  += lambda_dE' q (1 - u),  lambda_V[k+1] += lambda_dE' q u
//   lambda_dE     = lambda_dE'
//
// followed by lambda_p_t = A^T lambda_V (the same spectral kernel with
// conj(Z): the transpose of a circular convolution is the correlation)
// and the accumulation G += P_t conj(rfft(lambda_V)) from which the host
// forms dL/dZ and, by the chain rule, dL/d(R_s, f_r, Q).  Everything on the
// adjoint side runs in FP64; the forward keeps the engine's FP64 or
// F32P64 (float dE, FP64 phase and drift) arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "../../include/blond_b200.h"
#include "common.cuh"
#include "spectral.cuh"
#include "convolve.cuh"

namespace bb {

constexpr int kAdjThreads = 512;
constexpr int kAdjBlocks = 2;  // per SM
constexpr int kAdjMaxRf = 4;

struct AdjTurn {
    int64_t n;
    int n_rf;
    const double* V;   // this turn's n_rf amplitudes, frequencies, phases
    const double* om;
    const double* ph;
    double acc, charge, drift_c;
    const double* vind;  // S induced voltages of this turn, or nullptr
    int S;
    double bc0, inv_w;   // bin centres bc0 + k / inv_w
    int smem_hist;       // 1: block-private histograms in shared memory
    int fix_bits;        // fixed-point units per particle: 2^fix_bits
    double fix_scale;    // 2^fix_bits
    int vind_smem;       // 1: a copy of vind in shared memory for the gathers
};

template <int PREC> struct AdjE;
template <> struct AdjE<BLOND_PREC_F64> { using E = double; };
template <> struct AdjE<BLOND_PREC_F32P64> { using E = float; };

__device__ __forceinline__ double adj_reduce_2pi(double x) {
    const double inv2pi = 0.15915494309189533577;
    const double twopi = 6.28318530717958647692;
    return fma(-rint(x * inv2pi), twopi, x);
}

// Cloud-in-cell deposit of a unit weight at dt, in fixed point with 2^b
// units per particle: the weights are w1 = round(u 2^b) and w0 = 2^b - w1,
// accumulated with integer atomics, so every particle deposits exactly one
// unit and the profile does not depend on the order of the atomics (a run
// repeats bit for bit, which finite-difference checks of the map rely
// on).  b = min(52, 62 - ceil(log2(n + 1))) keeps n units below 2^63.
typedef unsigned long long u64;

inline int fixed_bits(int64_t n) {
    int lg = 0;
    while (lg < 63 && (1ull << lg) < (u64)n + 1) ++lg;
    return std::min(52, 62 - lg);
}

// (scale = 2^b: the product is exact, as ldexp's would be; floor(f) is the
// round-down conversion for the f > -1 that get here)
__device__ __forceinline__ void cic_deposit(u64* h, int S, double t, double bc0,
                                            double inv_w, int bits, double scale) {
    const double f = (t - bc0) * inv_w;
    if (!(f > -1.0 && f < (double)S)) return;  // also drops NaN
    const int j = __double2int_rd(f);
    const u64 w1 = (u64)__double2ll_rn((f - (double)j) * scale);
    const u64 w0 = (1ull << bits) - w1;
    if (j >= 0 && w0) atomicAdd(&h[j], w0);
    if (j + 1 < S && w1) atomicAdd(&h[j + 1], w1);
}

// The same deposit into a block's shared memory.  A 64-bit shared atomic is a
// compare-and-swap loop (forward turn of 2e6 particles 22 us with it, 11 us
// without a deposit), so the block keeps, per cell j (particles with floor(f)
// = j, slot j + 1), the count and the sum of w1 in two 32-bit words with the
// carry passed on: three native atomics.  flush_split forms the bins,
// sum w0 = count 2^b - sum w1, exactly as the 64-bit sums would.
struct SplitHist {
    unsigned *cnt, *lo, *hi;  // S + 1 slots each
};
__device__ __forceinline__ SplitHist split_hist(void* sh, int S) {
    unsigned* p = static_cast<unsigned*>(sh);
    return {p, p + (S + 1), p + 2 * (S + 1)};
}
__host__ __device__ inline size_t split_bytes(int S) {
    return (12 * (size_t)(S + 1) + 15) & ~(size_t)15;
}
__device__ __forceinline__ void zero_split(const SplitHist& h, int S) {
    for (int k = threadIdx.x; k < 3 * (S + 1); k += blockDim.x) h.cnt[k] = 0u;
}
__device__ __forceinline__ void split_deposit(const SplitHist& h, int S, double t, double bc0,
                                              double inv_w, double scale) {
    const double f = (t - bc0) * inv_w;
    if (!(f > -1.0 && f < (double)S)) return;  // also drops NaN
    const int j = __double2int_rd(f);
    const u64 w1 = (u64)__double2ll_rn((f - (double)j) * scale);
    const unsigned lo = (unsigned)w1;
    unsigned hi = (unsigned)(w1 >> 32);
    atomicAdd(&h.cnt[j + 1], 1u);
    const unsigned old = atomicAdd(&h.lo[j + 1], lo);
    if (old + lo < old) ++hi;
    if (hi) atomicAdd(&h.hi[j + 1], hi);
}
__device__ __forceinline__ void flush_split(const SplitHist& h, u64* g, int S, int bits) {
    for (int k = threadIdx.x; k < S; k += blockDim.x) {
        const u64 here = ((u64)h.hi[k + 1] << 32) + h.lo[k + 1];
        const u64 below = ((u64)h.hi[k] << 32) + h.lo[k];
        const u64 v = ((u64)h.cnt[k + 1] << bits) - here + below;
        if (v) atomicAdd(&g[k], v);
    }
}

__device__ __forceinline__ void flush_shared(const double* h, double* g, int S) {
    for (int k = threadIdx.x; k < S; k += blockDim.x)
        if (h[k] != 0.0) atomicAdd(&g[k], h[k]);
}

// The profile array is accumulated in place as fixed point (its zero bit
// pattern is 0.0) and converted to counts afterwards.
__global__ void fixed_to_counts_kernel(double* p, int S, int bits) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x)
        p[k] = ldexp((double)reinterpret_cast<const u64*>(p)[k], -bits);
}

__global__ void fixed_to_counts_from_kernel(const u64* raw, double* p, int S, int bits) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < S; k += gridDim.x * blockDim.x)
        p[k] = ldexp((double)raw[k], -bits);
}

__global__ void __launch_bounds__(kAdjThreads)
adj_deposit_kernel(const double* __restrict__ dt, int64_t n, int S, double bc0, double inv_w,
                   int smem_hist, int bits, u64* __restrict__ prof) {
    extern __shared__ __align__(16) unsigned char shq[];
    const SplitHist h = split_hist(shq, S);
    if (smem_hist) zero_split(h, S);
    __syncthreads();
    const double scale = ldexp(1.0, bits);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (smem_hist) split_deposit(h, S, dt[i], bc0, inv_w, scale);
        else cic_deposit(prof, S, dt[i], bc0, inv_w, bits, scale);
    }
    __syncthreads();
    if (smem_hist) flush_split(h, prof, S, bits);
}

// Converts the fixed-point profile to counts in the block that finishes
// last (a counter in global memory, reset by that block), so a turn needs
// no separate conversion launch.  Every block calls it after its own
// deposits; no block waits on another.
__device__ void convert_when_last(u64* prof, int S, int bits, unsigned* done) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = threadIdx.x; k < S; k += blockDim.x)
        reinterpret_cast<double*>(prof)[k] = ldexp((double)__ldcg(prof + k), -bits);
    if (threadIdx.x == 0) *done = 0u;
}

// One turn of one particle, as the forward map takes it (vind may be null).
template <int PREC, int NRF>
__device__ __forceinline__ void adj_step(double& t, typename AdjE<PREC>::E& e, const AdjTurn& T,
                                         const double* vind, const double* sV, const double* sOm,
                                         const double* sPh, double acc, double drift_c) {
    using E = typename AdjE<PREC>::E;
    const double q = T.charge;
    if (vind) {
        const double f = (t - T.bc0) * T.inv_w;
        if (f >= 0.0 && f < (double)(T.S - 1)) {
            const int k = __double2int_rd(f);
            const double w = f - (double)k;
            e += (E)(q * (vind[k] * (1.0 - w) + vind[k + 1] * w));
        }
    }
    if (PREC == BLOND_PREC_F64) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NRF; ++j) s += sV[j] * sin(fma(sOm[j], t, sPh[j]));
        e += (E)(q * s + acc);
    } else {
        // the engine's F32P64 sine: reduction in double, polynomial in float
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < NRF; ++j) s += (float)sV[j] * rf_sinf(fma(sOm[j], t, sPh[j]));
        e += (E)q * s + (E)acc;
    }
    t = t + drift_c * (double)e;
}

// NRF: the number of RF harmonics, a template parameter so that every
// harmonic's arithmetic is issued only when it exists (a runtime count
// under an unrolled loop to kAdjMaxRf left the unused harmonics' sines
// issued under predicates).
template <int PREC, int NRF>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks)
adj_forward_kernel(const AdjTurn T, const double* dt_in, const void* dE_in, double* dt_out,
                   void* dE_out, u64* prof_out, unsigned* done) {
    using E = typename AdjE<PREC>::E;
    // launched with programmatic stream serialization inside the runs: the
    // next grid may launch now; the programme and shared memory are set up
    // before this grid waits for the one before it
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char shf[];
    __shared__ double sV[kAdjMaxRf], sOm[kAdjMaxRf], sPh[kAdjMaxRf];
    if (threadIdx.x < T.n_rf) {
        sV[threadIdx.x] = T.V[threadIdx.x];
        sOm[threadIdx.x] = T.om[threadIdx.x];
        sPh[threadIdx.x] = T.ph[threadIdx.x];
    }
    const bool dep = prof_out != nullptr;
    const bool hsm = dep && T.smem_hist;
    const SplitHist h = split_hist(shf, T.S);
    if (hsm) zero_split(h, T.S);
    pdl_wait();  // coordinates, induced voltage and counter of the grids before
    const double* vind = T.vind;
    if (vind && T.vind_smem) {
        double* sv = reinterpret_cast<double*>(shf + (hsm ? split_bytes(T.S) : 0));
        for (int k = threadIdx.x; k < T.S; k += blockDim.x) sv[k] = T.vind[k];
        vind = sv;
    }
    __syncthreads();
    const E* dEi = static_cast<const E*>(dE_in);
    E* dEo = static_cast<E*>(dE_out);
    // the next two particles are on their way while one is computed
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double t1 = i < T.n ? dt_in[i] : 0.0, t2 = i + stride < T.n ? dt_in[i + stride] : 0.0;
    E e1 = i < T.n ? dEi[i] : E(0), e2 = i + stride < T.n ? dEi[i + stride] : E(0);
    for (; i < T.n; i += stride) {
        double t = t1;
        E e = e1;
        t1 = t2;
        e1 = e2;
        if (i + 2 * stride < T.n) {
            t2 = dt_in[i + 2 * stride];
            e2 = dEi[i + 2 * stride];
        }
        adj_step<PREC, NRF>(t, e, T, vind, sV, sOm, sPh, T.acc, T.drift_c);
        dt_out[i] = t;
        dEo[i] = e;
        if (hsm) split_deposit(h, T.S, t, T.bc0, T.inv_w, T.fix_scale);
        else if (dep) cic_deposit(prof_out, T.S, t, T.bc0, T.inv_w, T.fix_bits, T.fix_scale);
    }
    if (hsm) {
        __syncthreads();
        flush_split(h, prof_out, T.S, T.fix_bits);
    }
    if (dep && done) convert_when_last(prof_out, T.S, T.fix_bits, done);
}

// The turn-start coordinates of up to kAdjSegTurns turns of a segment: with
// their induced voltages stored, nothing couples the particles, so R of a
// thread stay in registers for all the turns and only dt is written each turn
// (states[q] at the start of turn q, states[n_sub] at the end).  Bound: those
// writes, 8 B per particle and turn (2e6 particles: 2.5 us a turn; one pass
// per turn took 11).  Each turn's voltages come to shared memory two turns
// ahead (three buffers, one barrier a turn).  The same operations as
// adj_forward_kernel, so the same bits.
constexpr int kAdjSegTurns = 64;
constexpr int kAdjSegThreads = 512;

struct AdjSegment {
    AdjTurn T;
    int n_sub;
    const double* vind;  // [n_sub][S] or nullptr
    int smem_vind;
    double acc[kAdjSegTurns], drift_c[kAdjSegTurns];
};

__device__ __forceinline__ void adj_copy8(double* smem, const double* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

template <int PREC, int NRF, int R>
__global__ void __launch_bounds__(kAdjSegThreads, 2)
adj_segment_kernel(const AdjSegment G, const double* dt_in, const void* dE_in, double* states,
                   void* dE_out) {
    using E = typename AdjE<PREC>::E;
    extern __shared__ double shv[];
    __shared__ double sV[kAdjSegTurns][kAdjMaxRf], sOm[kAdjSegTurns][kAdjMaxRf],
        sPh[kAdjSegTurns][kAdjMaxRf];
    const AdjTurn& T = G.T;
    const int S = T.S;
    for (int x = threadIdx.x; x < G.n_sub * T.n_rf; x += blockDim.x) {
        const int q = x / T.n_rf, j = x - q * T.n_rf;
        sV[q][j] = T.V[x];
        sOm[q][j] = T.om[x];
        sPh[q][j] = T.ph[x];
    }
    const E* const ein = static_cast<const E*>(dE_in);
    E* const eout = static_cast<E*>(dE_out);
    const bool staged = G.vind && G.smem_vind;
    auto stage = [&](int q) {
        if (q < G.n_sub)
            for (int k = threadIdx.x; k < S; k += blockDim.x)
                adj_copy8(shv + (q % 3) * S + k, G.vind + (size_t)q * S + k);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int64_t tile = (int64_t)gridDim.x * blockDim.x;
    // every thread of a block runs the same tiles (the barriers need them)
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < T.n; i0 += R * tile) {
        double t[R];
        E e[R];
        const int64_t i = i0 + threadIdx.x;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool in = i + r * tile < T.n;
            t[r] = in ? dt_in[i + r * tile] : 0.0;
            e[r] = in ? ein[i + r * tile] : E(0);
            if (in) states[i + r * tile] = t[r];
        }
        __syncthreads();  // the programme, and the last tile's voltages are free
        if (staged) {
            stage(0);
            stage(1);
        }
        for (int q = 0; q < G.n_sub; ++q) {
            const double* v = G.vind ? G.vind + (size_t)q * S : nullptr;
            if (staged) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();
                stage(q + 2);  // into the buffer of turn q - 1
                v = shv + (q % 3) * S;
            }
            double* const out = states + (size_t)(q + 1) * T.n;
#pragma unroll
            for (int r = 0; r < R; ++r)
                adj_step<PREC, NRF>(t[r], e[r], T, v, sV[q], sOm[q], sPh[q], G.acc[q],
                                    G.drift_c[q]);
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (i + r * tile < T.n) out[i + r * tile] = t[r];
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (i + r * tile < T.n) eout[i + r * tile] = e[r];
    }
    if (staged) asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// accum[k] += sum_t P_t[k] conj(L_t[k]) over n_rows rows of M1 values.
__global__ void adj_accumulate_kernel(const double2* P, const double2* L, int64_t M1, int n_rows,
                                      double2* accum) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < M1;
         k += (int64_t)gridDim.x * blockDim.x) {
        double re = 0.0, im = 0.0;
        for (int t = n_rows - 1; t >= 0; --t) {
            const double2 p = P[t * M1 + k], l = L[t * M1 + k];
            re += p.x * l.x + p.y * l.y;
            im += p.y * l.x - p.x * l.y;
        }
        accum[k].x += re;
        accum[k].y += im;
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One backward turn (kick = 1), or only the deposit adjoint of a profile
// at dt_next (kick = 0).  Bound: latency and the shared FP64 additions
// (compare-and-swap loops, 10 of 34 us at 2e6 particles); prefetching the next
// particle and one gather per table took it from 37.5 us (50 cold).
template <int NRF>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks)
adj_backward_kernel(const AdjTurn T, int kick, const double* __restrict__ dt,
                    const double* __restrict__ dt_next, const double* __restrict__ lam_p_next,
                    double* __restrict__ lam_dt, double* __restrict__ lam_dE,
                    double* __restrict__ lam_v, double* __restrict__ grad_rf) {
    extern __shared__ double sh[];
    __shared__ double sV[kAdjMaxRf], sOm[kAdjMaxRf], sPh[kAdjMaxRf];
    __shared__ double red[kAdjThreads / 32][2 * kAdjMaxRf];
    const int S = T.S;
    const bool sm = T.smem_hist != 0;
    // shared memory: the deposit adjoint's slopes (cell j at j + 1), the
    // block's lambda_V, then the voltage's steps: one gather each a particle
    double* const slope = sh;
    double* lv = sm ? sh + S + 1 : lam_v;
    double* const step = sh + 2 * S + 1;
    const double q = T.charge;
    auto slope_at = [&](int j) {  // of cell j in [-1, S - 1]
        const double a = j >= 0 ? lam_p_next[j] : 0.0;
        const double b = j + 1 < S ? lam_p_next[j + 1] : 0.0;
        return (b - a) * T.inv_w;
    };
    pdl_launch_dependents();  // as in adj_forward_kernel
    if (kick && threadIdx.x < T.n_rf) {
        sV[threadIdx.x] = T.V[threadIdx.x];
        sOm[threadIdx.x] = T.om[threadIdx.x];
        sPh[threadIdx.x] = T.ph[threadIdx.x];
    }
    const bool steps = T.vind && T.vind_smem;
    if (sm)
        for (int k = threadIdx.x; k < S; k += blockDim.x) lv[k] = 0.0;
    if (steps)  // the voltages were stored by the forward run
        for (int k = threadIdx.x; k < S - 1; k += blockDim.x)
            step[k] = q * (T.vind[k + 1] - T.vind[k]);
    pdl_wait();  // the adjoint and coordinates of the grids before
    if (sm && lam_p_next)
        for (int k = threadIdx.x; k <= S; k += blockDim.x) slope[k] = slope_at(k - 1);
    __syncthreads();
    double gv[kAdjMaxRf], gp[kAdjMaxRf];
#pragma unroll
    for (int j = 0; j < kAdjMaxRf; ++j) gv[j] = gp[j] = 0.0;
    // the next particle's values are on their way while one is computed
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double n_ldt = 0.0, n_ldE = 0.0, n_t = 0.0, n_tn = 0.0;
    auto fetch = [&](int64_t x) {
        if (x < T.n) {
            n_ldt = lam_dt[x];
            n_ldE = lam_dE[x];
            if (kick) n_t = dt[x];
            if (lam_p_next) n_tn = dt_next[x];
        }
    };
    fetch(i);
    for (; i < T.n; i += stride) {
        double ldt = n_ldt, ldE = n_ldE;
        const double t = n_t, t_next = n_tn;
        fetch(i + stride);
        if (lam_p_next) {
            const double f = (t_next - T.bc0) * T.inv_w;
            if (f > -1.0 && f < (double)S) {
                const int j = __double2int_rd(f);
                ldt += sm ? slope[j + 1] : slope_at(j);
            }
        }
        if (kick) {
            const double lE = ldE + T.drift_c * ldt;
            double dg = 0.0;
#pragma unroll
            for (int j = 0; j < NRF; ++j) {
                // sin and cos at the forward's phase, to rounding (the
                // forward map itself keeps CUDA's sin)
                double s, c;
                rf_sincos(fma(sOm[j], t, sPh[j]), &s, &c);
                dg += sV[j] * sOm[j] * c;
                gv[j] += lE * s;
                gp[j] += lE * sV[j] * c;
            }
            dg *= q;
            if (T.vind) {
                const double f = (t - T.bc0) * T.inv_w;
                if (f >= 0.0 && f < (double)(S - 1)) {
                    const int k = __double2int_rd(f);
                    const double w = f - (double)k;
                    dg += (steps ? step[k] : q * (T.vind[k + 1] - T.vind[k])) * T.inv_w;
                    atomicAdd(&lv[k], lE * q * (1.0 - w));
                    atomicAdd(&lv[k + 1], lE * q * w);
                }
            }
            ldt += lE * dg;
            ldE = lE;
        }
        lam_dt[i] = ldt;
        lam_dE[i] = ldE;
    }
    if (kick) {
        // programme gradients: warp sums, then one atomic per block and value
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
        for (int j = 0; j < NRF; ++j) {
            const double a = warp_sum(gv[j]), b = warp_sum(gp[j]);
            if (lane == 0) {
                red[w][j] = a;
                red[w][kAdjMaxRf + j] = b;
            }
        }
        __syncthreads();
        if (threadIdx.x < 2 * T.n_rf) {
            const int j = threadIdx.x < T.n_rf ? threadIdx.x : kAdjMaxRf + threadIdx.x - T.n_rf;
            double s = 0.0;
            for (int r = 0; r < (int)(blockDim.x >> 5); ++r) s += red[r][j];
            atomicAdd(&grad_rf[threadIdx.x], q * s);
        }
        if (sm) flush_shared(lv, lam_v, S);
    }
}

static int adj_smem_limit() { return (device_info().max_smem_optin - 4096) / 16; }

// Shared memory a block may take for its copy of the induced voltage (with
// the arrays it holds anyway), so that kAdjBlocks still fit on an SM.
constexpr size_t kAdjVindSmem = 96 * 1024;
// Shared memory of adj_segment_kernel's three voltage buffers (two blocks per
// SM); longer profiles gather from global memory.
constexpr size_t kAdjSegSmem = 100 * 1024;

template <typename K>
static int adj_allow_smem(K kernel, bool* done) {
    const DeviceInfo& d = device_info();
    if (!done[d.device & 63]) {
        cudaFuncAttributes fa;
        BB_CUDA(cudaFuncGetAttributes(&fa, kernel));
        BB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     d.max_smem_optin - (int)fa.sharedSizeBytes));
        done[d.device & 63] = true;
    }
    return BLOND_OK;
}

// The same once per kernel and device, for kernels chosen at run time.
template <typename K>
static int adj_allow_smem(K kernel) {
    static std::mutex m;
    static std::set<std::pair<const void*, int>> done;
    const DeviceInfo& d = device_info();
    std::lock_guard<std::mutex> g(m);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), d.device);
    if (done.count(key)) return BLOND_OK;
    cudaFuncAttributes fa;
    BB_CUDA(cudaFuncGetAttributes(&fa, kernel));
    BB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 d.max_smem_optin - (int)fa.sharedSizeBytes));
    done.insert(key);
    return BLOND_OK;
}

// Launch, with programmatic stream serialization when pdl (the turn loops
// of the runs: each grid launches while the one before it finishes).
template <typename... KArgs, typename... Args>
static int adj_launch(void (*k)(KArgs...), int grid, size_t smem, cudaStream_t s, bool pdl,
                      Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kAdjThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    BB_CUDA(cudaLaunchKernelEx(&cfg, k, args...));
    return BLOND_OK;
}

// The kernels for the run-time harmonic count n_rf (0..kAdjMaxRf).
template <int PREC>
static auto adj_forward_for(int n_rf) {
    switch (n_rf) {
        case 0: return adj_forward_kernel<PREC, 0>;
        case 1: return adj_forward_kernel<PREC, 1>;
        case 2: return adj_forward_kernel<PREC, 2>;
        case 3: return adj_forward_kernel<PREC, 3>;
        default: return adj_forward_kernel<PREC, 4>;
    }
}

static auto adj_backward_for(int n_rf) {
    switch (n_rf) {
        case 0: return adj_backward_kernel<0>;
        case 1: return adj_backward_kernel<1>;
        case 2: return adj_backward_kernel<2>;
        case 3: return adj_backward_kernel<3>;
        default: return adj_backward_kernel<4>;
    }
}

// One forward turn.  With a counter (`done`, zero between launches) the
// last block converts the deposited profile to counts; without one a
// second launch does, unless the caller wants the fixed-point deposit (raw).
static int adj_forward_launch(int precision, const double* dt_in, const void* dE_in,
                              double* dt_out, void* dE_out, int64_t n, int n_rf,
                              const double* voltage, const double* omega_rf,
                              const double* phi_rf, double acc_kick, double charge,
                              double drift_coeff, const double* induced_voltage,
                              int n_slices, double bin_center0, double inv_bin_width,
                              double* profile_out, unsigned* done, void* stream,
                              bool pdl = false, bool raw = false) {
    BB_CHECK_ARG(precision == BLOND_PREC_F64 || precision == BLOND_PREC_F32P64,
                 "adjoint_forward_turn: unknown precision %d", precision);
    BB_CHECK_SIZE(n_rf >= 0 && n_rf <= kAdjMaxRf, "adjoint_forward_turn: n_rf=%d not in "
                  "[0, %d]", n_rf, kAdjMaxRf);
    BB_CHECK_ARG(n >= 0 && n_slices >= 2, "adjoint_forward_turn: bad size");
    BB_CHECK_ARG((n == 0 || (dt_in && dE_in && dt_out && dE_out)) &&
                     (n_rf == 0 || (voltage && omega_rf && phi_rf)),
                 "adjoint_forward_turn: null pointer");
    if (n == 0) return BLOND_OK;
    AdjTurn T = {};
    T.n = n;
    T.n_rf = n_rf;
    T.V = voltage;
    T.om = omega_rf;
    T.ph = phi_rf;
    T.acc = acc_kick;
    T.charge = charge;
    T.drift_c = drift_coeff;
    T.vind = induced_voltage;
    T.S = n_slices;
    T.bc0 = bin_center0;
    T.inv_w = inv_bin_width;
    T.smem_hist = n_slices <= adj_smem_limit() ? 1 : 0;
    T.fix_bits = fixed_bits(n);
    T.fix_scale = ldexp(1.0, T.fix_bits);
    const size_t hist = profile_out && T.smem_hist ? split_bytes(n_slices) : 0;
    T.vind_smem = induced_voltage && hist + sizeof(double) * n_slices <= kAdjVindSmem;
    const size_t smem = hist + (T.vind_smem ? sizeof(double) * n_slices : 0);
    const int grid = particle_grid(n, kAdjThreads, kAdjBlocks);
    cudaStream_t s = as_stream(stream);
    u64* prof = reinterpret_cast<u64*>(profile_out);
    int rc;
    const auto k = precision == BLOND_PREC_F64 ? adj_forward_for<BLOND_PREC_F64>(n_rf)
                                               : adj_forward_for<BLOND_PREC_F32P64>(n_rf);
    if ((rc = adj_allow_smem(k))) return rc;
    if ((rc = adj_launch(k, grid, smem, s, pdl, T, dt_in, dE_in, dt_out, dE_out, prof, done)))
        return rc;
    if (profile_out && !done && !raw) {
        fixed_to_counts_kernel<<<(n_slices + 255) / 256, 256, 0, s>>>(profile_out, n_slices,
                                                                      T.fix_bits);
        BB_LAUNCH_CHECK();
    }
    return BLOND_OK;
}

// One backward turn (blond_adjoint_backward_turn), with programmatic stream
// serialization when pdl.
static int adj_backward_launch(const double* dt, const double* dt_next, int64_t n,
                                double* lam_dt, double* lam_dE, const double* lam_p_next,
                                int kick, int n_rf, const double* voltage,
                                const double* omega_rf, const double* phi_rf, double charge,
                                double drift_coeff, const double* induced_voltage,
                                int n_slices, double bin_center0, double inv_bin_width,
                                double* lam_v, double* grad_rf, void* stream,
                                bool pdl = false) {
    BB_CHECK_SIZE(n_rf >= 0 && n_rf <= kAdjMaxRf, "adjoint_backward_turn: n_rf=%d not in "
                  "[0, %d]", n_rf, kAdjMaxRf);
    BB_CHECK_ARG(n >= 0 && n_slices >= 2, "adjoint_backward_turn: bad size");
    BB_CHECK_ARG(n == 0 || (lam_dt && lam_dE), "adjoint_backward_turn: null adjoint");
    BB_CHECK_ARG(!lam_p_next || dt_next, "adjoint_backward_turn: lam_p_next needs dt_next");
    BB_CHECK_ARG(!kick || ((n == 0 || dt) && grad_rf && (!induced_voltage || lam_v) &&
                           (n_rf == 0 || (voltage && omega_rf && phi_rf))),
                 "adjoint_backward_turn: null pointer");
    if (n == 0) return BLOND_OK;
    AdjTurn T = {};
    T.n = n;
    T.n_rf = n_rf;
    T.V = voltage;
    T.om = omega_rf;
    T.ph = phi_rf;
    T.charge = charge;
    T.drift_c = drift_coeff;
    T.vind = kick ? induced_voltage : nullptr;
    T.S = n_slices;
    T.bc0 = bin_center0;
    T.inv_w = inv_bin_width;
    T.smem_hist = n_slices <= adj_smem_limit() ? 1 : 0;
    T.vind_smem = T.vind && T.smem_hist && 3 * sizeof(double) * n_slices <= kAdjVindSmem;
    int rc;
    const auto k = adj_backward_for(kick ? n_rf : 0);
    if ((rc = adj_allow_smem(k))) return rc;
    const size_t smem =
        T.smem_hist ? sizeof(double) * ((T.vind_smem ? 3 : 2) * (size_t)n_slices + 1) : 0;
    const int grid = particle_grid(n, kAdjThreads, kAdjBlocks);
    return adj_launch(k, grid, smem, as_stream(stream), pdl, T, kick, dt, dt_next, lam_p_next,
                      lam_dt, lam_dE, lam_v, grad_rf);
}

// Fixed-point deposit of dt into prof (added to what it holds).
static int adj_deposit_launch(const double* dt, int64_t n, int n_slices, double bin_center0,
                              double inv_bin_width, u64* prof, cudaStream_t s) {
    static bool done[64] = {false};
    int rc;
    if ((rc = adj_allow_smem(adj_deposit_kernel, done))) return rc;
    const int sm = n_slices <= adj_smem_limit() ? 1 : 0;
    const int grid = particle_grid(n, kAdjThreads, kAdjBlocks);
    adj_deposit_kernel<<<grid, kAdjThreads, sm ? split_bytes(n_slices) : 0, s>>>(
        dt, n, n_slices, bin_center0, inv_bin_width, sm, fixed_bits(n), prof);
    BB_LAUNCH_CHECK();
    return BLOND_OK;
}

}  // namespace bb

using namespace bb;

extern "C" {

int blond_adjoint_deposit(const double* dt, int64_t n, int n_slices, double bin_center0,
                          double inv_bin_width, double* profile, void* stream) {
    BB_CHECK_ARG(n >= 0 && n_slices >= 1, "adjoint_deposit: bad size");
    BB_CHECK_ARG(profile && (n == 0 || dt), "adjoint_deposit: null pointer");
    if (n == 0) return BLOND_OK;
    cudaStream_t s = as_stream(stream);
    const int rc = adj_deposit_launch(dt, n, n_slices, bin_center0, inv_bin_width,
                                      reinterpret_cast<u64*>(profile), s);
    if (rc) return rc;
    fixed_to_counts_kernel<<<(n_slices + 255) / 256, 256, 0, s>>>(profile, n_slices,
                                                                  fixed_bits(n));
    BB_LAUNCH_CHECK();
    return BLOND_OK;
}

int blond_adjoint_forward_turn(int precision, const double* dt_in, const void* dE_in,
                               double* dt_out, void* dE_out, int64_t n, int n_rf,
                               const double* voltage, const double* omega_rf,
                               const double* phi_rf, double acc_kick, double charge,
                               double drift_coeff, const double* induced_voltage,
                               int n_slices, double bin_center0, double inv_bin_width,
                               double* profile_out, void* stream) {
    return adj_forward_launch(precision, dt_in, dE_in, dt_out, dE_out, n, n_rf, voltage,
                              omega_rf, phi_rf, acc_kick, charge, drift_coeff,
                              induced_voltage, n_slices, bin_center0, inv_bin_width,
                              profile_out, nullptr, stream);
}

int blond_adjoint_backward_turn(const double* dt, const double* dt_next, int64_t n,
                                double* lam_dt, double* lam_dE, const double* lam_p_next,
                                int kick, int n_rf, const double* voltage,
                                const double* omega_rf, const double* phi_rf, double charge,
                                double drift_coeff, const double* induced_voltage,
                                int n_slices, double bin_center0, double inv_bin_width,
                                double* lam_v, double* grad_rf, void* stream) {
    return adj_backward_launch(dt, dt_next, n, lam_dt, lam_dE, lam_p_next, kick, n_rf, voltage,
                               omega_rf, phi_rf, charge, drift_coeff, induced_voltage, n_slices,
                               bin_center0, inv_bin_width, lam_v, grad_rf, stream);
}

int blond_adjoint_spectral(int mode, const double* x, int n_slices, const double* impedance,
                           int64_t n_fft, double scale, double* y, double* spectrum,
                           double* accum, void* stream) {
    BB_CHECK_ARG(mode == 0 || mode == 1, "adjoint_spectral: mode must be 0 or 1");
    BB_CHECK_ARG(x && impedance && y && n_slices >= 1, "adjoint_spectral: bad argument");
    BB_CHECK_ARG(mode == 0 || (spectrum && accum), "adjoint_spectral: mode 1 needs the "
                 "stored spectrum and the accumulator");
    SpecParams P = {};
    if (!make_spec_plan(n_fft, P.p)) {
        set_error("adjoint_spectral: n_fft=%lld is not an even 5-smooth length <= %lld",
                  (long long)n_fft, (long long)kMaxClusterFFT);
        return BLOND_ERR_UNSUPPORTED;
    }
    P.mode = SPEC_FORWARD | SPEC_MULTIPLY | SPEC_INVERSE;
    P.in_f64 = x;
    P.n_in = n_slices;
    P.H = reinterpret_cast<const double2*>(impedance);
    P.out = y;
    P.n_out = n_slices < n_fft ? n_slices : n_fft;
    P.out_scale = -scale / (double)P.p.M;
    if (mode == 0 && spectrum) {
        P.mode |= SPEC_OUT_SPECTRUM;
        P.spec_out = reinterpret_cast<double2*>(spectrum);
    }
    if (mode == 1) {
        P.mode |= SPEC_ACCUM;
        P.acc_a = reinterpret_cast<const double2*>(spectrum);
        P.acc_g = reinterpret_cast<double2*>(accum);
    }
    return launch_spectral(P, as_stream(stream));
}

}  // extern "C"

namespace bb {

// Scratch of a run, ordered on its stream: no device synchronisation, and
// calls of other threads and streams have their own.  The library's pool
// keeps at most 64 MB of freed scratch per device and returns the rest.
static cudaMemPool_t adj_pool() {
    static cudaMemPool_t pool[64] = {nullptr};
    static std::mutex mu;
    const int dev = device_info().device;
    std::lock_guard<std::mutex> lock(mu);
    if (!pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        uint64_t keep = 64ull << 20;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        pool[dev] = p;
    }
    return pool[dev];
}

struct AdjScratch {
    void* p = nullptr;
    cudaStream_t s = nullptr;
    ~AdjScratch() {
        if (p) cudaFreeAsync(p, s);
    }
    int init(size_t bytes, cudaStream_t stream) {
        const cudaMemPool_t pool = adj_pool();
        if (!pool) {
            set_error("adjoint run: memory pool creation failed");
            return BLOND_ERR_CUDA;
        }
        s = stream;
        BB_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool, stream));
        return BLOND_OK;
    }
};

// The induced voltages of a run: short profiles by direct convolution
// (convolve.cuh) -- then the spectra follow in one batched transform after
// the turn loop -- others by one transform per turn.  One plan, twiddle table
// and response for the whole run.
struct AdjVoltage {
    SpecPlan plan = {};
    ConvPlan cplan = {};
    bool conv = false;
    AdjScratch mem;
    double2* tw = nullptr;
    double* hx = nullptr;
    u64* raw = nullptr;      // fixed-point profile between two turns
    int* ticket = nullptr;
    unsigned* done = nullptr;
    double2* rows = nullptr;  // spectra of kRows profiles
    static constexpr int kRows = 64;

    // H: the run's impedance or nullptr (then only `done` is set up)
    int init(const double* H, int64_t n_fft, int S, cudaStream_t s) {
        size_t tw_bytes = 0, y_bytes = 0, hx_bytes = 0, row_bytes = 0;
        int rc;
        if (H) {
            if (!make_spec_plan(n_fft, plan)) {
                set_error("adjoint run: n_fft=%lld is not an even 5-smooth length <= %lld",
                          (long long)n_fft, (long long)kMaxClusterFFT);
                return BLOND_ERR_UNSUPPORTED;
            }
            if ((rc = prepare_spectral())) return rc;
            conv = n_fft >= S && make_conv_plan(S, n_fft, 1, cplan);
            if (conv && (rc = prepare_conv())) return rc;
            tw_bytes = (spec_twiddle_bytes(plan) + 15) & ~(size_t)15;
            if (conv) {
                y_bytes = 8 * ((size_t)n_fft + 1);
                hx_bytes = 16 * (size_t)S;
                row_bytes = 16 * (size_t)kRows * (n_fft / 2 + 1);
            }
        }
        const size_t raw_bytes = (8 * (size_t)S + 15) & ~(size_t)15;
        y_bytes = (y_bytes + 15) & ~(size_t)15;
        if ((rc = mem.init(tw_bytes + y_bytes + hx_bytes + row_bytes + raw_bytes + 16, s)))
            return rc;
        char* p = static_cast<char*>(mem.p);
        tw = reinterpret_cast<double2*>(p);
        rows = reinterpret_cast<double2*>(p + tw_bytes);
        double* const y = reinterpret_cast<double*>(p + tw_bytes + row_bytes);
        hx = reinterpret_cast<double*>(p + tw_bytes + row_bytes + y_bytes);
        raw = reinterpret_cast<u64*>(p + tw_bytes + row_bytes + y_bytes + hx_bytes);
        ticket = reinterpret_cast<int*>(reinterpret_cast<char*>(raw) + raw_bytes);
        done = reinterpret_cast<unsigned*>(ticket + 1);
        BB_CUDA(cudaMemsetAsync(raw, 0, raw_bytes + 16, s));
        if (H && (rc = fill_spec_twiddles(plan, tw, s))) return rc;
        if (conv && (rc = conv_response_async(reinterpret_cast<const double2*>(H), n_fft, S, y,
                                              hx, s)))
            return rc;
        return BLOND_OK;
    }
    // y = -scale h (*) x of one profile: counts, or with `deposit` the
    // fixed-point one in `raw`, which is converted to counts and cleared
    int convolve(const double* x, int fix_bits, double* counts, int S, double scale, double* y,
                 cudaStream_t s) const {
        ConvParams P = {};
        P.p = cplan;
        P.hx = hx;
        P.in_f64 = x;
        if (!x) {
            P.in_fix = raw;
            P.fix_unit = ldexp(1.0, -fix_bits);
            P.profile_out = counts;
            P.ticket = ticket;
        }
        P.out = y;
        P.out_scale = -scale;
        P.pdl = 1;
        return launch_conv(P, s);
    }
    // spectra of n_rows consecutive profiles
    int spectra(const double* x, int S, int n_rows, double* out, cudaStream_t s) const {
        SpecParams P = {};
        shrink_spec_plan(plan, n_rows >= 64 ? 1 : 4, P.p);
        if (P.p.smem > device_info().max_smem_optin) P.p = plan;
        P.twg = tw;
        P.mode = SPEC_FORWARD | SPEC_OUT_SPECTRUM;
        P.in_f64 = x;
        P.n_in = S;
        P.spec_out = reinterpret_cast<double2*>(out);
        P.batch = n_rows;
        return launch_spectral(P, s);
    }
    // the same transform as blond_adjoint_spectral(mode, ...)
    int run(int mode, const double* x, int S, const double* H, double scale, double* y,
            double* spectrum, double* accum, cudaStream_t s) const {
        SpecParams P = {};
        P.p = plan;
        P.twg = tw;
        P.pdl = 1;  // inside the turn loops of the runs
        P.mode = SPEC_FORWARD | SPEC_MULTIPLY | SPEC_INVERSE;
        P.in_f64 = x;
        P.n_in = S;
        P.H = reinterpret_cast<const double2*>(H);
        P.out = y;
        P.n_out = S < plan.N ? S : plan.N;
        P.out_scale = -scale / (double)plan.M;
        if (mode == 0 && spectrum) {
            P.mode |= SPEC_OUT_SPECTRUM;
            P.spec_out = reinterpret_cast<double2*>(spectrum);
        }
        if (mode == 1) {
            P.mode |= SPEC_ACCUM;
            P.acc_a = reinterpret_cast<const double2*>(spectrum);
            P.acc_g = reinterpret_cast<double2*>(accum);
        }
        return launch_spectral(P, s);
    }
};

template <int PREC, int R>
static auto adj_segment_for(int n_rf) {
    switch (n_rf) {
        case 0: return adj_segment_kernel<PREC, 0, R>;
        case 1: return adj_segment_kernel<PREC, 1, R>;
        case 2: return adj_segment_kernel<PREC, 2, R>;
        case 3: return adj_segment_kernel<PREC, 3, R>;
        default: return adj_segment_kernel<PREC, 4, R>;
    }
}

// The turn-start coordinates of turns [0, n_sub) from dt_in, dE_in: states
// (n_sub + 1 rows) and the final energies.
static int launch_segment(int precision, const AdjSegment& G, const double* dt_in,
                          const void* dE_in, double* states, void* dE_out, cudaStream_t s) {
    // one particle a thread while that fills the SMs, else four
    const int64_t resident = (int64_t)device_info().sm_count * 2 * kAdjSegThreads;
    const bool one = G.T.n <= resident;
    const auto k = precision == BLOND_PREC_F64
                       ? (one ? adj_segment_for<BLOND_PREC_F64, 1>(G.T.n_rf)
                              : adj_segment_for<BLOND_PREC_F64, 4>(G.T.n_rf))
                       : (one ? adj_segment_for<BLOND_PREC_F32P64, 1>(G.T.n_rf)
                              : adj_segment_for<BLOND_PREC_F32P64, 4>(G.T.n_rf));
    int rc;
    if ((rc = adj_allow_smem(k))) return rc;
    const int grid = particle_grid(G.T.n, kAdjSegThreads, 2);
    const size_t smem = G.vind && G.smem_vind ? 3 * sizeof(double) * (size_t)G.T.S : 0;
    k<<<grid, kAdjSegThreads, smem, s>>>(G, dt_in, dE_in, states, dE_out);
    BB_LAUNCH_CHECK();
    return BLOND_OK;
}

}  // namespace bb

extern "C" {

int blond_adjoint_forward_run(int precision, double* dt, void* dE, int64_t n, int n_rf,
                              int64_t n_turns, const double* voltage, const double* omega_rf,
                              const double* phi_rf, const double* acc_kick,
                              const double* drift_coeff, double charge,
                              const double* impedance, int64_t n_fft, double scale,
                              double* induced_voltage, double* spectrum, double* profile,
                              int n_slices, double bin_center0, double inv_bin_width,
                              int checkpoint_every, double* ckpt_dt, void* ckpt_dE,
                              void* stream) {
    BB_CHECK_ARG(precision == BLOND_PREC_F64 || precision == BLOND_PREC_F32P64,
                 "adjoint_forward_run: precision must be F64 or F32P64");
    BB_CHECK_ARG(n >= 1 && n_turns >= 1 && n_slices >= 2 && checkpoint_every >= 1,
                 "adjoint_forward_run: bad size");
    BB_CHECK_ARG(dt && dE && voltage && omega_rf && phi_rf && acc_kick && drift_coeff &&
                     profile && ckpt_dt && ckpt_dE,
                 "adjoint_forward_run: null pointer");
    BB_CHECK_ARG(!impedance || (induced_voltage && spectrum),
                 "adjoint_forward_run: an impedance needs the induced-voltage and spectrum "
                 "arrays");
    cudaStream_t s = as_stream(stream);
    const size_t esz = precision == BLOND_PREC_F64 ? sizeof(double) : sizeof(float);
    const int64_t M1 = n_fft / 2 + 1;
    AdjVoltage sp;
    int rc;
    if ((rc = sp.init(impedance, n_fft, n_slices, s))) return rc;
    const int bits = fixed_bits(n);
    if (sp.conv) {
        if ((rc = adj_deposit_launch(dt, n, n_slices, bin_center0, inv_bin_width, sp.raw, s)))
            return rc;
    } else if ((rc = blond_adjoint_deposit(dt, n, n_slices, bin_center0, inv_bin_width, profile,
                                           stream))) {
        return rc;
    }
    for (int64_t t = 0; t < n_turns; ++t) {
        if (t % checkpoint_every == 0) {
            const int64_t seg = t / checkpoint_every;
            BB_CUDA(cudaMemcpyAsync(ckpt_dt + seg * n, dt, sizeof(double) * n,
                                    cudaMemcpyDeviceToDevice, s));
            BB_CUDA(cudaMemcpyAsync(static_cast<char*>(ckpt_dE) + (size_t)seg * n * esz, dE,
                                    esz * n, cudaMemcpyDeviceToDevice, s));
        }
        double* vind = impedance ? induced_voltage + t * n_slices : nullptr;
        double* const next = profile + (t + 1) * n_slices;
        if (sp.conv)
            rc = sp.convolve(nullptr, bits, profile + t * n_slices, n_slices, scale, vind, s);
        else if (impedance)
            rc = sp.run(0, profile + t * n_slices, n_slices, impedance, scale, vind,
                        spectrum + t * M1 * 2, nullptr, s);
        if (rc) return rc;
        // (with the convolution the next turn's launch converts the deposit)
        if ((rc = adj_forward_launch(
                 precision, dt, dE, dt, dE, n, n_rf, voltage + t * n_rf, omega_rf + t * n_rf,
                 phi_rf + t * n_rf, acc_kick[t], charge, drift_coeff[t], vind, n_slices,
                 bin_center0, inv_bin_width, sp.conv ? reinterpret_cast<double*>(sp.raw) : next,
                 sp.conv ? nullptr : sp.done, stream, true, sp.conv)))
            return rc;
    }
    if (sp.conv) {
        fixed_to_counts_from_kernel<<<(n_slices + 255) / 256, 256, 0, s>>>(
            sp.raw, profile + n_turns * n_slices, n_slices, bits);
        BB_LAUNCH_CHECK();
        // the spectra of the turns' profiles, in launches of at most 4096
        for (int64_t t = 0; t < n_turns; t += 4096)
            if ((rc = sp.spectra(profile + t * n_slices, n_slices,
                                 (int)std::min<int64_t>(4096, n_turns - t),
                                 spectrum + t * M1 * 2, s)))
                return rc;
    }
    return BLOND_OK;
}

int blond_adjoint_backward_run(int precision, int64_t n, int n_rf, int64_t n_turns,
                               const double* voltage, const double* omega_rf,
                               const double* phi_rf, const double* acc_kick,
                               const double* drift_coeff, double charge,
                               const double* impedance_conj, int64_t n_fft, double scale,
                               const double* induced_voltage, const double* spectrum,
                               int n_slices, double bin_center0, double inv_bin_width,
                               int checkpoint_every, const double* ckpt_dt,
                               const void* ckpt_dE, double* states, void* dE_work,
                               double* lam_dt, double* lam_dE, const double* lam_p_final,
                               double* lam_v, double* lam_pt, double* grad_rf,
                               double* spectrum_accum, void* stream) {
    BB_CHECK_ARG(precision == BLOND_PREC_F64 || precision == BLOND_PREC_F32P64,
                 "adjoint_backward_run: precision must be F64 or F32P64");
    BB_CHECK_ARG(n >= 1 && n_turns >= 1 && n_slices >= 2 && checkpoint_every >= 1,
                 "adjoint_backward_run: bad size");
    BB_CHECK_ARG(voltage && omega_rf && phi_rf && acc_kick && drift_coeff && ckpt_dt &&
                     ckpt_dE && states && dE_work && lam_dt && lam_dE && grad_rf,
                 "adjoint_backward_run: null pointer");
    BB_CHECK_ARG(!impedance_conj || (induced_voltage && spectrum && lam_v && lam_pt &&
                                     spectrum_accum),
                 "adjoint_backward_run: an impedance needs the stored induced voltages and "
                 "spectra and the adjoint arrays");
    cudaStream_t s = as_stream(stream);
    const size_t esz = precision == BLOND_PREC_F64 ? sizeof(double) : sizeof(float);
    const int64_t M1 = n_fft / 2 + 1;
    const int64_t K = checkpoint_every;
    const int64_t nseg = (n_turns + K - 1) / K;
    const bool has_z = impedance_conj != nullptr;
    AdjVoltage sp;
    int rc;
    if (has_z && (rc = sp.init(impedance_conj, n_fft, n_slices, s))) return rc;
    const double* lam_p = lam_p_final;
    for (int64_t seg = nseg - 1; seg >= 0; --seg) {
        const int64_t a = seg * K, b = std::min(n_turns, (seg + 1) * K);
        // the segment's turn-start coordinates, recomputed from its checkpoint
        for (int64_t t = a; t < b; t += kAdjSegTurns) {
            AdjSegment G = {};
            G.T.n = n;
            G.T.n_rf = n_rf;
            G.T.V = voltage + t * n_rf;
            G.T.om = omega_rf + t * n_rf;
            G.T.ph = phi_rf + t * n_rf;
            G.T.charge = charge;
            G.T.S = n_slices;
            G.T.bc0 = bin_center0;
            G.T.inv_w = inv_bin_width;
            G.n_sub = (int)std::min<int64_t>(kAdjSegTurns, b - t);
            G.vind = has_z ? induced_voltage + t * n_slices : nullptr;
            G.smem_vind = 3 * sizeof(double) * n_slices <= kAdjSegSmem;
            for (int q = 0; q < G.n_sub; ++q) {
                G.acc[q] = acc_kick[t + q];
                G.drift_c[q] = drift_coeff[t + q];
            }
            const bool first = t == a;
            if ((rc = launch_segment(
                     precision, G, first ? ckpt_dt + seg * n : states + (t - a) * n,
                     first ? static_cast<const void*>(static_cast<const char*>(ckpt_dE) +
                                                      (size_t)seg * n * esz)
                           : dE_work,
                     states + (t - a) * n, dE_work, s)))
                return rc;
        }
        for (int64_t t = b - 1; t >= a; --t) {
            if ((rc = adj_backward_launch(
                     states + (t - a) * n, states + (t - a + 1) * n, n, lam_dt, lam_dE, lam_p, 1,
                     n_rf, voltage + t * n_rf, omega_rf + t * n_rf, phi_rf + t * n_rf, charge,
                     drift_coeff[t], has_z ? induced_voltage + t * n_slices : nullptr,
                     n_slices, bin_center0, inv_bin_width,
                     has_z ? lam_v + t * n_slices : nullptr, grad_rf + t * 2 * n_rf, stream,
                     true)))
                return rc;
            if (has_z) {
                if (sp.conv)
                    rc = sp.convolve(lam_v + t * n_slices, 0, nullptr, n_slices, scale,
                                     lam_pt + t * n_slices, s);
                else
                    rc = sp.run(1, lam_v + t * n_slices, n_slices, impedance_conj, scale,
                                lam_pt + t * n_slices,
                                const_cast<double*>(spectrum) + t * M1 * 2, spectrum_accum, s);
                if (rc) return rc;
                lam_p = lam_pt + t * n_slices;
            } else {
                lam_p = nullptr;
            }
        }
        // the impedance's gradient from the segment's spectra
        for (int64_t hi = b; sp.conv && hi > a; hi -= AdjVoltage::kRows) {
            const int64_t lo = std::max(a, hi - AdjVoltage::kRows);
            const int rows = (int)(hi - lo);
            if ((rc = sp.spectra(lam_v + lo * n_slices, n_slices, rows,
                                 reinterpret_cast<double*>(sp.rows), s)))
                return rc;
            adj_accumulate_kernel<<<(int)((M1 + 127) / 128), 128, 0, s>>>(
                reinterpret_cast<const double2*>(spectrum) + lo * M1, sp.rows, M1, rows,
                reinterpret_cast<double2*>(spectrum_accum));
            BB_LAUNCH_CHECK();
        }
    }
    // the turn-0 profile is a deposit of the initial dt
    if (lam_p)
        return blond_adjoint_backward_turn(nullptr, ckpt_dt, n, lam_dt, lam_dE, lam_p, 0, n_rf,
                                           nullptr, nullptr, nullptr, charge, 0.0, nullptr,
                                           n_slices, bin_center0, inv_bin_width, nullptr,
                                           nullptr, stream);
    return BLOND_OK;
}

}  // extern "C"
