// Direct circular convolution head: see convolve.cuh.
#include "convolve.cuh"
#include "spectral.cuh"

#include <algorithm>

namespace bb {

// dst[q] = load(q) for q < n, eight loads of a thread in flight at a time.
template <typename F>
__device__ __forceinline__ void fill_shared(double* dst, int n, int tid, int nth, F load) {
    constexpr int U = 8;
    for (int q0 = tid; q0 < n; q0 += U * nth) {
        decltype(load(0)) v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = q0 + u * nth < n ? load(q0 + u * nth) : 0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (q0 + u * nth < n) dst[q0 + u * nth] = (double)v[u];
    }
}

// Each thread keeps kConvTile outputs and walks one contiguous segment of
// the profile: the outputs need kConvTile consecutive values of hx, and the
// next bin needs the same ones moved by one, so a step is two shared loads
// (one new response value, one bin) for kConvTile multiply-adds.  A segment
// has an odd length, so the 32 segments of a warp fall on different banks.
//
// One more warp takes what the outputs do not wait for: the converted
// profile, the beam-phase sums, the ticket that tells when every block has
// read the histogram, then (last block) the clearing and the loop's turn.  On
// a computing warp the ticket's round trip alone took 0.7 us of a 4 us launch.
// The loop is one chain of memory round trips, the longest of the launch: its
// sums are taken from the histogram itself while the other warps load, and the
// blocks' sums are fetched while the histogram is cleared (turns of 2e4
// particles, 2000 slices 13.0 -> 11.8 us; 10.9 without the loop).
template <bool FB>
__global__ void __launch_bounds__(kConvThreads + 32)
conv_head_kernel(const ConvParams P, const typename ConvLoopArg<FB>::type fb) {
    pdl_launch_dependents();
    extern __shared__ double csm[];
    __shared__ double red[kConvThreads / 32][kConvTile];
    __shared__ double vs[kConvTile * kConvMaxGroups];
    const int S = P.p.S, g = P.p.groups, L = P.p.seg, wpg = P.p.wpg;
    const int T = 32 * wpg * L, nth = 32 * wpg * g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int beam = P.batch ? (int)blockIdx.x / P.p.ctas : 0;
    const int cta = (int)blockIdx.x - beam * P.p.ctas;
    const int i0 = cta * P.p.chunk;
    const int n_own = min(P.p.chunk, S - i0);
    const int64_t boff = (int64_t)beam * S;
    double* const prof = csm;     // T bins, zero beyond S
    double* const hw = csm + T;   // the responses of this block's outputs
    const int nh = T + kConvTile * g - 1;

    // hw[q] multiplies bin j of output i0 + o at q = o - j + T - 1
    const double* const hx = P.hx + (int64_t)beam * (2 * S - 1);
    fill_shared(hw, nh, tid, nth + 32, [&](int q) {
        const int x = i0 + q - (T - S);
        return x >= 0 && x < 2 * S - 1 ? __ldg(hx + x) : 0.0;
    });
    pdl_wait();  // the particle pass: histogram, turn counter, RF programme
    const long long turn = P.turn ? *P.turn : 0;
    if constexpr (FB) {
        // this block's bins of the beam-phase sums, while the others load
        if (tid >= nth) {
            double s = 0.0, c = 0.0;
            if (turn >= fb.delay) {
                const FbBins b = fb_bins(fb, turn);
                for (int o = lane; o < n_own; o += 32)
                    fb_add<true>(b, i0 + o,
                                 P.in_i32 ? (double)__ldcg(P.in_i32 + i0 + o)
                                          : __ldcg(P.in_f64 + i0 + o),
                                 s, c);
            }
            for (int d = 16; d > 0; d >>= 1) {
                s += __shfl_down_sync(0xffffffffu, s, d);
                c += __shfl_down_sync(0xffffffffu, c, d);
            }
            if (lane == 0) {
                fb.phase_partials[2 * cta] = s;
                fb.phase_partials[2 * cta + 1] = c;
            }
        }
    }
    // with the loop the extra warp leaves the profile to the others: reading it
    // too, after its sums, held the block barrier back (0.5 us of a turn at 200
    // to 9000 slices)
    const int nfill = FB ? nth : nth + 32;
    const int end = tid < nfill ? T : 0;
    if (P.in_i32) {
        const int* const in = P.in_i32 + boff;
        fill_shared(prof, end, tid, nfill, [&](int j) { return j < S ? __ldcg(in + j) : 0; });
    } else if (P.in_fix) {
        const unsigned long long* const in = P.in_fix + boff;
        fill_shared(prof, end, tid, nfill, [&](int j) {
            return j < S ? (double)__ldcg(in + j) * P.fix_unit : 0.0;
        });
    } else {
        const double* const in = P.in_f64 + boff;
        fill_shared(prof, end, tid, nfill, [&](int j) { return j < S ? __ldcg(in + j) : 0.0; });
    }
    __syncthreads();
    if (tid >= nth) {
        if (P.profile_out)
            for (int o = lane; o < n_own; o += 32) P.profile_out[boff + i0 + o] = prof[i0 + o];
        if (!P.ticket) return;
        int last = 0;
        if (lane == 0) {
            __threadfence();
            last = atomicAdd(P.ticket + beam, 1) == P.p.ctas - 1;
        }
        if (!__shfl_sync(0xffffffffu, last, 0)) return;
        __threadfence();
        // the blocks' sums, on their way while the histogram is cleared
        constexpr int kSums = 5;  // at most 148 blocks
        double ps[kSums], pc[kSums];
        if constexpr (FB) {
#pragma unroll
            for (int k = 0; k < kSums; ++k) {
                const int q = lane + 32 * k;
                ps[k] = q < P.p.ctas ? __ldcg(fb.phase_partials + 2 * q) : 0.0;
                pc[k] = q < P.p.ctas ? __ldcg(fb.phase_partials + 2 * q + 1) : 0.0;
            }
        }
        // every block has read the histogram and the counter
        if (P.in_i32)
            for (int j = lane; j < S; j += 32) P.in_i32[boff + j] = 0;
        if (P.in_fix)
            for (int j = lane; j < S; j += 32) P.in_fix[boff + j] = 0ull;
        if (lane == 0) {
            P.ticket[beam] = 0;
            if (P.turn && beam == 0) *P.turn = turn + 1;
        }
        if constexpr (FB) {
            double s = 0.0, c = 0.0;
#pragma unroll
            for (int k = 0; k < kSums; ++k) {
                s += ps[k];
                c += pc[k];
            }
            for (int q = lane + 32 * kSums; q < P.p.ctas; q += 32) {
                s += __ldcg(fb.phase_partials + 2 * q);
                c += __ldcg(fb.phase_partials + 2 * q + 1);
            }
            for (int d = 16; d > 0; d >>= 1) {
                s += __shfl_down_sync(0xffffffffu, s, d);
                c += __shfl_down_sync(0xffffffffu, c, d);
            }
            if (lane == 0) fb_turn_end(fb, turn, s, c, 0.0);
        }
        return;
    }

    const int grp = warp / wpg, seg = (warp - grp * wpg) * 32 + lane;
    const double* const pj = prof + seg * L;
    const double* const hj = hw + (T - 1 - seg * L + kConvTile * grp);
    double acc[kConvTile], w[kConvTile];
#pragma unroll
    for (int r = 0; r < kConvTile; ++r) {
        acc[r] = 0.0;
        w[r] = r ? hj[r] : 0.0;
    }
    // response r of step u sits in w[(r - u) mod kConvTile]
    auto step = [&](int j, int u) {
        w[(kConvTile - u) % kConvTile] = hj[-(j + u)];
        const double x = pj[j + u];
#pragma unroll
        for (int r = 0; r < kConvTile; ++r)
            acc[r] = fma(w[(r + kConvTile - u) % kConvTile], x, acc[r]);
    };
    int j = 0;
    for (; j + kConvTile <= L; j += kConvTile) {
#pragma unroll
        for (int u = 0; u < kConvTile; ++u) step(j, u);
    }
#pragma unroll
    for (int u = 0; u < kConvTile - 1; ++u)
        if (j + u < L) step(j, u);
    // sums over the warp's segments: each exchange halves the outputs a lane
    // still carries
#pragma unroll
    for (int h = 16, c = kConvTile / 2; c >= 1; h >>= 1, c >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int r = 0; r < c; ++r) {
            const double send = up ? acc[r] : acc[r + c];
            const double keep = up ? acc[r + c] : acc[r];
            acc[r] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    if ((lane & 3) == 0) red[warp][lane >> 2] = acc[0];
    // the computing warps' barrier
    auto compute_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nth) : "memory"); };
    compute_sync();

    if (tid < kConvTile * g) {
        double v = 0.0;
        for (int q = 0; q < wpg; ++q) v += red[(tid / kConvTile) * wpg + q][tid % kConvTile];
        const int i = i0 + tid;
        v *= P.beam_scale ? P.beam_scale[beam] : P.out_scale;
        if (i < S) {
            if (P.ind_coeff) {
                // np.gradient(profile, dbc): central inside, one-sided at ends
                double d;
                if (i == 0) d = (prof[1] - prof[0]) / P.ind_dbc;
                else if (i == S - 1) d = (prof[S - 1] - prof[S - 2]) / P.ind_dbc;
                else d = (prof[i + 1] - prof[i - 1]) / (2.0 * P.ind_dbc);
                v = v + P.ind_coeff[turn] * d;
            }
            if (tid < n_own) P.out[boff + i] = v;
            if (P.interp) {
                long long t = turn < 0 ? 0 : turn;
                if (t >= P.n_turns) t = P.n_turns - 1;
                double s = 0.0;
                for (int j = 0; j < P.n_rf; ++j)
                    s += P.rf_v[t * P.n_rf + j] *
                         rf_sin(P.rf_om[t * P.n_rf + j] * P.bc[i] + P.rf_ph[t * P.n_rf + j]);
                v = s + v;  // rf_voltage + induced_voltage
            }
        }
        vs[tid] = v;
    }
    if (P.table) {
        compute_sync();
        if (tid < n_own && i0 + tid < S - 1) {
            const int n = i0 + tid;
            const double a0 = vs[tid], a1 = vs[tid + 1];
            const double inv_w = P.beam_inv_w ? P.beam_inv_w[beam] : P.inv_w;
            double acc_t = 0.0;
            if (P.interp) {
                long long t = turn < 0 ? 0 : turn;
                if (t >= P.n_turns) t = P.n_turns - 1;
                acc_t = P.acc[t];
            }
            if (!P.table_f32) {
                const double b = P.bc[boff + n];
                reinterpret_cast<double2*>(P.table)[boff + n] =
                    P.interp ? lik_entry(a0, a1, b, P.charge, inv_w, acc_t)
                             : lik_entry0(a0, a1, b, P.charge, inv_w);
            } else {
                reinterpret_cast<float2*>(P.table)[boff + n] =
                    P.interp ? make_float2((float)(P.charge * a0 + acc_t),
                                           (float)(P.charge * (a1 - a0) * inv_w))
                             : make_float2((float)(P.charge * a0),
                                           (float)(P.charge * (a1 - a0) * inv_w));
            }
        }
    }
}

bool make_conv_plan(int S, int64_t N, int B, ConvPlan& plan) {
    if (S < 2) return false;
    const int sms = device_info().sm_count;
    const bool pow2 = (N & (N - 1)) == 0;
    // one profile: S^2 multiply-adds over all SMs against the FFT's chain of
    // phases (turns of 2e4 particles, FFT -> convolution: 201 slices 16.9 ->
    // 7.2 us, 1000 19.8 -> 7.8, 2000 24.1 -> 8.6, 4096 13.2 -> 9.9, 8192
    // 12.8 -> 14.2, 9000 61.6 -> 16.2)
    if (B == 1 && pow2 && S > 4600) return false;
    // a batch: the profiles' multiply-adds share the SMs (37 beams of 400
    // slices 21.2 -> 14.5 us a turn, but 64 of 512 would be 16 -> 23 and 256 of
    // 300 37 -> 40); up to 8 beams of up to 4600 slices convolve as single ones
    // do.  A beam of a batch has the single-beam engine's bits where both
    // convolve; elsewhere the batch takes spectral_kernel and the single beam
    // may take another head (9000 slices: convolution; 8192 and 14000: the
    // 16-CTA transform; 512 in a batch of 64: convolution), and the voltages
    // agree within the two heads' rounding, 4e-14 of the largest.
    if (B > 1 && (int64_t)B * S * S > 8'000'000 && (B > 8 || S > 4600)) return false;
    int g = 1;
    while (g < kConvMaxGroups && (kConvTile * g - 1) * sms < S) ++g;
    if ((kConvTile * g - 1) * sms < S) return false;
    // segments of the profile, from S alone: a sum's order, hence its bits,
    // is the same in a batch as for a single beam
    plan.wpg = g <= 4 ? 4 : (g <= 8 ? 2 : 1);
    // a batch that fills the SMs takes more outputs per block
    while (B > 1 && 32 * plan.wpg * (g + 1) <= kConvThreads && g < kConvMaxGroups &&
           (int64_t)B * ((S + kConvTile * g - 2) / (kConvTile * g - 1)) > 8 * sms)
        ++g;
    plan.S = S;
    plan.groups = g;
    plan.chunk = kConvTile * g - 1;
    plan.ctas = (S + plan.chunk - 1) / plan.chunk;
    const int nseg = 32 * plan.wpg;
    plan.seg = ((S + nseg - 1) / nseg) | 1;
    plan.smem = (int)sizeof(double) * (2 * nseg * plan.seg + kConvTile * g - 1);
    return plan.smem + 8192 <= device_info().max_smem_optin;
}

// hx[b][x] = y[b][(x - (S - 1)) mod N]
__global__ void conv_response_kernel(const double* y, int64_t N, int S, int B, double* hx) {
    for (int64_t b = blockIdx.y; b < B; b += gridDim.y)
        for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < 2 * S - 1;
             x += (int64_t)gridDim.x * blockDim.x) {
            int64_t d = x - (S - 1);
            if (d < 0) d += N;
            hx[b * (2 * S - 1) + x] = y[b * N + d];
        }
}
// A grid has at most 65535 rows: more beams than that share them.
static dim3 response_grid(int S, int B) {
    return dim3((2 * S + 254) / 256, std::min(B, 65535));
}

int make_conv_response(const double2* H, int64_t N, int S, int B, double** hx) {
    *hx = nullptr;
    double* y = nullptr;
    BB_CUDA(cudaMalloc((void**)&y, sizeof(double) * (size_t)N * B));
    int rc = BLOND_OK;
    for (int b = 0; b < B && rc == BLOND_OK; ++b)
        rc = blond_irfft_f64(reinterpret_cast<const double*>(H + (size_t)b * (N / 2 + 1)), N,
                             y + (size_t)b * N, N, nullptr);
    if (rc == BLOND_OK && cudaMalloc((void**)hx, sizeof(double) * (size_t)(2 * S - 1) * B) !=
                              cudaSuccess) {
        set_error("convolution head: cudaMalloc failed");
        rc = BLOND_ERR_CUDA;
    }
    if (rc == BLOND_OK) {
        conv_response_kernel<<<response_grid(S, B), 256>>>(y, N, S, B, *hx);
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
            set_error("convolution head: response kernel failed");
            rc = BLOND_ERR_CUDA;
        }
    }
    cudaFree(y);
    if (rc && *hx) {
        cudaFree(*hx);
        *hx = nullptr;
    }
    return rc;
}

int conv_response_async(const double2* H, int64_t N, int S, double* y, double* hx,
                        cudaStream_t stream) {
    const int rc = blond_irfft_f64(reinterpret_cast<const double*>(H), N, y, N, stream);
    if (rc) return rc;
    conv_response_kernel<<<response_grid(S, 1), 256, 0, stream>>>(y, N, S, 1, hx);
    BB_LAUNCH_CHECK();
    return BLOND_OK;
}

int prepare_conv() {
    static bool done[64] = {false};
    const DeviceInfo& d = device_info();
    if (!done[d.device & 63]) {
        BB_CUDA(cudaFuncSetAttribute(conv_head_kernel<false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     d.max_smem_optin - 8192));
        BB_CUDA(cudaFuncSetAttribute(conv_head_kernel<true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     d.max_smem_optin - 8192));
        done[d.device & 63] = true;
    }
    return BLOND_OK;
}

template <bool FB>
static int launch_conv_t(const ConvParams& P, const typename ConvLoopArg<FB>::type& fb,
                         cudaStream_t stream) {
    int rc = prepare_conv();
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P.p.ctas * (P.batch > 0 ? P.batch : 1));
    cfg.blockDim = dim3(32 * P.p.wpg * P.p.groups + 32);
    cfg.dynamicSmemBytes = P.p.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = P.pdl ? 1 : 0;
    BB_CUDA(cudaLaunchKernelEx(&cfg, conv_head_kernel<FB>, P, fb));
    return BLOND_OK;
}

int launch_conv(const ConvParams& P, cudaStream_t stream) {
    return launch_conv_t<false>(P, ConvNoLoop{}, stream);
}

int launch_conv_loop(const ConvParams& P, const FeedbackArgs& fb, cudaStream_t stream) {
    return launch_conv_t<true>(P, fb, stream);
}

}  // namespace bb
