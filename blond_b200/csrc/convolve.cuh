// The induced voltage of a short profile as a direct circular convolution.
//
//     V = -scale irfft(Z rfft(p, N))[:S]   (impedances/impedance.py:457-489)
//
// is the product of p with a circulant matrix, V_i = -scale sum_{j < S}
// h_{(i - j) mod N} p_j with h = irfft(Z): S^2 multiply-adds, every output
// independent of the others.  The FFT head (spectral.cuh) does far fewer
// operations, but as a chain of about fifteen dependent phases in one
// cluster, each a barrier and a shared-memory round trip: 13 to 15 us a
// launch even at 200 slices, where nothing else on the GPU runs.  Here every
// SM computes its own outputs from the whole profile in one phase: no
// barrier between blocks, no exchange (a block forms the one voltage beyond
// its range again, so that the interpolation-table entries need no
// neighbour), and h is fetched before the wait for the particle pass.
//
// Bound: latency up to about 2000 slices (one read of the histogram from L2,
// one block reduction), FP64 issue beyond (S^2 / (148 SMs x 64 per clock)).
#pragma once

#include "common.cuh"
#include "feedback.cuh"

namespace bb {

constexpr int kConvThreads = 512;   // computing threads, at most; one more warp
                                    // clears up and runs the loop
constexpr int kConvTile = 8;        // outputs a thread accumulates in registers
constexpr int kConvMaxGroups = 12;  // tiles of outputs per block

struct ConvPlan {
    int S = 0;       // slices: inputs and outputs
    int groups = 0;  // tiles of kConvTile outputs per block
    int wpg = 0;     // warps per tile: 32 wpg segments of the profile
    int chunk = 0;   // outputs a block owns: kConvTile groups - 1
    int ctas = 0;    // blocks per profile
    int seg = 0;     // profile bins per thread (odd: no bank conflicts)
    int smem = 0;
};

struct ConvParams {
    ConvPlan p;
    // the impulse response around 0: hx[B][2 S - 1], hx[x] = h_{(x - (S-1)) mod N}
    const double* hx;
    // the profile: exactly one of in_f64, in_i32 (the engine's histogram) and
    // in_fix (the adjoint's fixed-point deposit, 2^fix_bits units a particle);
    // the last two are zeroed by the last block to have read them
    const double* in_f64;
    int* in_i32;
    unsigned long long* in_fix;
    double fix_unit;          // 2^-fix_bits
    double* profile_out;      // the converted histogram or deposit
    double* out;              // the induced voltage
    double out_scale;
    const double* beam_scale; // batch: per profile, in place of out_scale
    // inductive impedance: out += ind_coeff[turn] gradient(profile)
    const double* ind_coeff;
    double ind_dbc;
    // interpolation table over the voltages (see SpecParams)
    void* table;
    int table_f32;
    double charge, inv_w;
    const double* beam_inv_w; // batch: per profile, in place of inv_w
    const double* bc;
    // interpolated tracker: the table holds the RF voltage at the bin
    // centres, the induced voltage and the acceleration kick
    int interp;
    const double* rf_v;
    const double* rf_om;
    const double* rf_ph;
    const double* acc;
    int n_rf;
    long long n_turns;
    long long* turn;          // device turn counter, advanced once
    int* ticket;              // one per profile, zero between launches (in_i32,
                              // in_fix, turn or a loop need it)
    int batch;                // profiles (0: one)
    int pdl;
};

struct ConvNoLoop {};
template <bool FB> struct ConvLoopArg { using type = ConvNoLoop; };
template <> struct ConvLoopArg<true> { using type = FeedbackArgs; };

// True when the direct convolution of B profiles of S slices is faster than
// the FFT of length N; then plan describes it.
bool make_conv_plan(int S, int64_t N, int B, ConvPlan& plan);
// hx (cudaMalloc'd, B (2 S - 1) doubles) from the impedances H, B x (N/2 + 1)
// values on the device.  Synchronous.
int make_conv_response(const double2* H, int64_t N, int S, int B, double** hx);
// The same on a stream into caller memory: hx and y (N doubles of scratch).
int conv_response_async(const double2* H, int64_t N, int S, double* y, double* hx,
                        cudaStream_t stream);
// Kernel attributes, set outside stream capture.
int prepare_conv();
int launch_conv(const ConvParams& P, cudaStream_t stream);
// With the beam-phase loop inside (single profile).
int launch_conv_loop(const ConvParams& P, const FeedbackArgs& fb, cudaStream_t stream);

}  // namespace bb
