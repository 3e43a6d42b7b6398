// Induced voltage of a long profile, n_fft a power of two:
//     out = scale irfft(Z rfft(profile))   (+ inductive term, table)
// as spectral_kernel computes it (packed real input of M = M1 x M2 complex
// points, four-step transform over a cluster of 16 CTAs), organised around
// what bounds it: the number of cluster-wide rounds and of dependent steps in
// each.  spectral_kernel takes four cluster barriers, reads every transposed
// element from another CTA's shared memory after the barrier, and walks
// interleaved transforms at a stride that puts a warp's accesses on one bank.
// Here
//   * a CTA owns rows k1 and M1 - k1 together, so the spectral step, which
//     pairs the bins k and M - k, needs no other CTA: two barriers, not four;
//   * transposed elements are pushed into the CTA that needs them before the
//     barrier, so that the next step reads its own shared memory;
//   * the forward transforms leave their output in bit-reversed order and the
//     inverse ones start from it: no permutation; the partner of position p
//     of row k1 sits at M2 - 1 - p of row M1 - k1;
//   * each transform is one warp's registers, stored contiguously with one
//     element of padding: no bank conflicts;
//   * the lengths are template parameters: no index division, small code.
#define BB_SPECTRAL_KERNELS
#include "head_fft.cuh"

namespace bb {

namespace {

constexpr int kHeadCtas = 16;

// The 32 P points of one transform across a warp: element lane + 32 q in
// v[q].  Forward: decimation in frequency, natural order in, bit-reversed
// out.  tw[q] = exp(-2 pi i q / L).
template <int P>
__device__ __forceinline__ void warp_dif(double2 (&v)[P], const double2* __restrict__ tw) {
    const int lane = threadIdx.x & 31;
    constexpr int L = 32 * P;
#pragma unroll
    for (int hq = P / 2; hq >= 1; hq >>= 1) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
            if (q & hq) continue;
            const double2 w = tw[((lane + 32 * q) & (32 * hq - 1)) * (L / (64 * hq))];
            const double2 x = v[q], y = v[q + hq];
            v[q] = cadd(x, y);
            v[q + hq] = cmul(csub(x, y), w);
        }
    }
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
        const double2 w = tw[(lane & (h - 1)) * (L / (2 * h))];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            double2 o;
            o.x = __shfl_xor_sync(0xffffffffu, v[q].x, h);
            o.y = __shfl_xor_sync(0xffffffffu, v[q].y, h);
            v[q] = up ? cmul(csub(o, v[q]), w) : cadd(v[q], o);
        }
    }
}

// Inverse (unscaled): decimation in time, bit-reversed order in, natural out.
template <int P>
__device__ __forceinline__ void warp_dit(double2 (&v)[P], const double2* __restrict__ tw) {
    const int lane = threadIdx.x & 31;
    constexpr int L = 32 * P;
#pragma unroll
    for (int h = 1; h <= 16; h <<= 1) {
        const bool up = (lane & h) != 0;
        const double2 w = cconj(tw[(lane & (h - 1)) * (L / (2 * h))]);
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const double2 t = up ? cmul(v[q], w) : v[q];
            double2 o;
            o.x = __shfl_xor_sync(0xffffffffu, t.x, h);
            o.y = __shfl_xor_sync(0xffffffffu, t.y, h);
            v[q] = up ? csub(o, t) : cadd(t, o);
        }
    }
#pragma unroll
    for (int hq = 1; hq < P; hq <<= 1) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
            if (q & hq) continue;
            const double2 w = cconj(tw[((lane + 32 * q) & (32 * hq - 1)) * (L / (64 * hq))]);
            const double2 x = v[q], y = cmul(v[q + hq], w);
            v[q] = cadd(x, y);
            v[q + hq] = csub(x, y);
        }
    }
}

__host__ __device__ constexpr int log2i(int x) { return x <= 1 ? 0 : 1 + log2i(x / 2); }

template <int P1, int P2>
struct HeadShape {
    static constexpr int M1 = 32 * P1, M2 = 32 * P2, M = M1 * M2;
    static constexpr int Bc = M2 / kHeadCtas, Br = M1 / kHeadCtas, per = M / kHeadCtas;
    static constexpr int ldc = M1 + 1, ldr = M2 + 1;  // padded transforms
    static constexpr int lgM1 = log2i(M1), lgM2 = log2i(M2);
    // the two-level tables' split, as make_spec_plan chooses it
    static constexpr int lgL = (lgM1 + lgM2 + 1) / 2, L = 1 << lgL, nA = (M + L - 1) / L;
    static constexpr int tw_count = M1 + M2 + 2 * nA + 2 * L;
    // bytes: columns, rows (at the end the voltages), twiddles, impedance and
    // the neighbour's voltages
    static constexpr int o_rows = 16 * Bc * ldc, o_tw = o_rows + 16 * Br * ldr,
                         o_h = o_tw + 16 * tw_count, o_nbr = o_h + 16 * (per + 1),
                         bytes = o_nbr + 8 * M1;
    static_assert(Br >= 2 && Bc >= 1, "16 CTAs");
};

// k1 of this CTA's row r and, for a k1, its CTA and row: rows q and M1 - q
// side by side, q = 0 paired with M1 / 2.
template <int M1, int Br>
__device__ __forceinline__ int row_k1(int c, int r) {
    const int q = c * (Br / 2) + (r >> 1);
    return q == 0 ? (r & 1) * (M1 / 2) : ((r & 1) ? M1 - q : q);
}
template <int M1, int Br>
__device__ __forceinline__ void row_owner(int k1, int& c, int& r) {
    const bool high = k1 >= M1 / 2;
    const int q = (k1 & (M1 / 2 - 1)) == 0 ? 0 : (high ? M1 - k1 : k1);
    c = q / (Br / 2);
    r = 2 * (q % (Br / 2)) + (high ? 1 : 0);
}

template <int P1, int P2>
__global__ void __launch_bounds__(kSpecThreads, 1)
head_fft_kernel(const SpecParams P) {
    using Sh = HeadShape<P1, P2>;
    constexpr int M1 = Sh::M1, M2 = Sh::M2, M = Sh::M, Bc = Sh::Bc, Br = Sh::Br;
    constexpr int nth = kSpecThreads, nw = nth / 32;
    cg::cluster_group cluster = cg::this_cluster();
    pdl_launch_dependents();
    const int c = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ __align__(16) unsigned char hsm[];
    double2* const cols = reinterpret_cast<double2*>(hsm);
    double2* const rows = reinterpret_cast<double2*>(hsm + Sh::o_rows);
    double2* const tw1 = reinterpret_cast<double2*>(hsm + Sh::o_tw);
    double2* const tw2 = tw1 + M1;
    double2* const tam = tw2 + M2;
    double2* const tbm = tam + Sh::nA;
    double2* const tan_ = tbm + Sh::L;
    double2* const tbn = tan_ + Sh::nA;
    double2* const hk = reinterpret_cast<double2*>(hsm + Sh::o_h);
    double2* const vloc = rows;  // per <= Br (M2 + 1) values, free by then
    double* const nbr = reinterpret_cast<double*>(hsm + Sh::o_nbr);
    // every CTA of the cluster runs (its shared memory may be written) once
    // this barrier, waited for before the first push, has completed
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

    if (P.twg) {
        for (int q = tid; q < Sh::tw_count; q += nth) cp_async16(&tw1[q], &P.twg[q]);
    } else {
        fill_twiddles(P.p, tw1, tw2, tam, tbm, tan_, tbn, tid, nth);
    }
    // the impedance of bin k1 + M1 k2 at [row][position of k2]
    for (int e = tid; e < Br * M2; e += nth) {
        const int r = e / M2, pos = e % M2;
        const int k2 = (int)(__brev((unsigned)pos) >> (32 - Sh::lgM2));
        cp_async16(&hk[e], &P.H[row_k1<M1, Br>(c, r) + M1 * k2]);
    }
    if (c == 0 && tid == 0) cp_async16(&hk[Br * M2], &P.H[M]);
    asm volatile("cp.async.commit_group;" ::: "memory");
    pdl_wait();  // the previous grid's histogram, counter and programme
    const long long turn = P.turn ? *P.turn : 0;
    const double ind = P.ind_coeff ? P.ind_coeff[turn] : 0.0;

    auto twm = [&](int j) { return cmul(tam[j >> Sh::lgL], tbm[j & (Sh::L - 1)]); };
    auto twn = [&](int j) { return cmul(tan_[j >> Sh::lgL], tbn[j & (Sh::L - 1)]); };

    // ---- columns n2 in [c Bc, (c + 1) Bc): z[m] = x[2m] + i x[2m+1], m = n2 + M2 n1
    {
        constexpr int U = Sh::per / nth >= 8 ? 8 : (Sh::per / nth >= 1 ? Sh::per / nth : 1);
        const int64_t nlim = P.n_in < (int64_t)2 * M ? P.n_in : (int64_t)2 * M;
        for (int e0 = tid; e0 < Sh::per; e0 += U * nth) {
            double2 x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * nth;
                const int64_t i = 2 * (int64_t)(c * Bc + e % Bc + M2 * (e / Bc));
                x[u] = make_double2(0.0, 0.0);
                if (P.in_i32) {
                    if (i < nlim) x[u].x = (double)__ldcg(P.in_i32 + i);
                    if (i + 1 < nlim) x[u].y = (double)__ldcg(P.in_i32 + i + 1);
                } else if (P.in_f32) {
                    if (i < nlim) x[u].x = (double)__ldcg(P.in_f32 + i);
                    if (i + 1 < nlim) x[u].y = (double)__ldcg(P.in_f32 + i + 1);
                } else {
                    if (i < nlim) x[u].x = __ldcg(P.in_f64 + i);
                    if (i + 1 < nlim) x[u].y = __ldcg(P.in_f64 + i + 1);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * nth;
                const int64_t i = 2 * (int64_t)(c * Bc + e % Bc + M2 * (e / Bc));
                cols[(e % Bc) * Sh::ldc + e / Bc] = x[u];
                if (P.in_i32) {
                    if (i < nlim) P.in_i32[i] = 0;
                    if (i + 1 < nlim) P.in_i32[i + 1] = 0;
                    if (P.profile_out) {
                        if (i < nlim) P.profile_out[i] = x[u].x;
                        if (i + 1 < nlim) P.profile_out[i + 1] = x[u].y;
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

    // ---- column transforms, the four-step twiddle W_M^(n2 k1), each element
    // to its row's CTA
    for (int b = warp; b < Bc; b += nw) {
        double2 v[P1];
#pragma unroll
        for (int q = 0; q < P1; ++q) v[q] = cols[b * Sh::ldc + lane + 32 * q];
        warp_dif<P1>(v, tw1);
        const int n2 = c * Bc + b;
#pragma unroll
        for (int q = 0; q < P1; ++q) {
            const int k1 = (int)(__brev((unsigned)(lane + 32 * q)) >> (32 - Sh::lgM1));
            int oc, r;
            row_owner<M1, Br>(k1, oc, r);
            cluster.map_shared_rank(rows, oc)[r * Sh::ldr + n2] = cmul(v[q], twm(n2 * k1));
        }
    }
    cluster.sync();
    // ---- row transforms
    for (int r = warp; r < Br; r += nw) {
        double2 v[P2];
#pragma unroll
        for (int q = 0; q < P2; ++q) v[q] = rows[r * Sh::ldr + lane + 32 * q];
        warp_dif<P2>(v, tw2);
#pragma unroll
        for (int q = 0; q < P2; ++q) rows[r * Sh::ldr + lane + 32 * q] = v[q];
    }
    __syncthreads();
    // ---- the bins k and M - k: spectrum of the real input, x Z, and back to
    // the packed form of the real output
    const int items = (Br / 2) * M2 + (c == 0 ? 1 : 0);
    for (int e = tid; e < items; e += nth) {
        int ra, pa, rb, pb;  // rows and positions of k and M - k
        if (c == 0 && e <= M2) {
            if (e <= M2 / 2) {  // row k1 = 0: k2 = e and M2 - e
                ra = rb = 0;
                pa = (int)(__brev((unsigned)e) >> (32 - Sh::lgM2));
                pb = (int)(__brev((unsigned)((M2 - e) & (M2 - 1))) >> (32 - Sh::lgM2));
            } else {  // row M1 / 2
                ra = rb = 1;
                pa = 2 * (e - M2 / 2 - 1);  // even positions: k2 < M2 / 2
                pb = M2 - 1 - pa;
            }
        } else {
            const int x = c == 0 ? e - 1 : e;
            ra = 2 * (x / M2);
            rb = ra + 1;
            pa = x % M2;
            pb = M2 - 1 - pa;
        }
        const int ia = ra * Sh::ldr + pa, ib = rb * Sh::ldr + pb;
        const double2 Za = rows[ia], Zb = rows[ib];
        const double2 Ha = hk[ra * M2 + pa], Hb = hk[rb * M2 + pb];
        if (c == 0 && e == 0) {
            // X[0] and X[M] are real; irfft ignores their products' imaginary parts
            const double y0 = (Za.x + Za.y) * Ha.x, ym = (Za.x - Za.y) * hk[Br * M2].x;
            rows[ia] = make_double2(0.5 * (y0 + ym), 0.5 * (y0 - ym));
            continue;
        }
        const int k = row_k1<M1, Br>(c, ra) +
                      M1 * (int)(__brev((unsigned)pa) >> (32 - Sh::lgM2));
        const double2 w = twn(k);
        const double2 E = cscale(cadd(Za, cconj(Zb)), 0.5);
        const double2 wO = cmul(w, crot<false>(cscale(csub(Za, cconj(Zb)), 0.5)));
        const double2 Ya = cmul(cadd(E, wO), Ha);          // X[k] Z[k]
        const double2 Yb = cmul(cconj(csub(E, wO)), Hb);   // X[M-k] Z[M-k]
        const double2 Ye = cscale(cadd(Ya, cconj(Yb)), 0.5);
        const double2 Yo = cmul(cconj(w), cscale(csub(Ya, cconj(Yb)), 0.5));
        rows[ia] = cadd(Ye, crot<true>(Yo));
        if (ib != ia) rows[ib] = cadd(cconj(Ye), crot<true>(cconj(Yo)));
    }
    __syncthreads();
    // ---- inverse row transforms, the conjugate twiddle, each element to its
    // column's CTA at the position its transform starts from
    for (int r = warp; r < Br; r += nw) {
        double2 v[P2];
#pragma unroll
        for (int q = 0; q < P2; ++q) v[q] = rows[r * Sh::ldr + lane + 32 * q];
        warp_dit<P2>(v, tw2);
        const int k1 = row_k1<M1, Br>(c, r);
        const int at = (int)(__brev((unsigned)k1) >> (32 - Sh::lgM1));
#pragma unroll
        for (int q = 0; q < P2; ++q) {
            const int m2 = lane + 32 * q;
            cluster.map_shared_rank(cols, m2 / Bc)[(m2 % Bc) * Sh::ldc + at] =
                cmul(v[q], cconj(twm(k1 * m2)));
        }
    }
    cluster.sync();
    // ---- inverse column transforms: y[2m], y[2m+1] with m = n2 + M2 m1
    const int64_t S = P.n_in;
    auto value = [&](int64_t n, double y) {
        double v = y * P.out_scale;
        if (P.ind_coeff) {
            // np.gradient(profile, dbc): central inside, one-sided at ends
            const double* const p = P.profile_out ? P.profile_out : P.in_f64;
            double d;
            if (S < 2 || n >= S) d = 0.0;
            else if (n == 0) d = (p[1] - p[0]) / P.ind_dbc;
            else if (n == S - 1) d = (p[S - 1] - p[S - 2]) / P.ind_dbc;
            else d = (p[n + 1] - p[n - 1]) / (2.0 * P.ind_dbc);
            v = v + ind * d;
        }
        return v;
    };
    for (int b = warp; b < Bc; b += nw) {
        double2 v[P1];
#pragma unroll
        for (int q = 0; q < P1; ++q) v[q] = cols[b * Sh::ldc + lane + 32 * q];
        warp_dit<P1>(v, tw1);
#pragma unroll
        for (int q = 0; q < P1; ++q) {
            const int m1 = lane + 32 * q;
            const int64_t n = 2 * (int64_t)(c * Bc + b + M2 * m1);
            const double2 o = make_double2(value(n, v[q].x), value(n + 1, v[q].y));
            if (P.out_f32) {
                if (n < P.n_out) P.out_f32[n] = (float)o.x;
                if (n + 1 < P.n_out) P.out_f32[n + 1] = (float)o.y;
            } else {
                if (n < P.n_out) P.out[n] = o.x;
                if (n + 1 < P.n_out) P.out[n + 1] = o.y;
            }
            if (P.table) {
                vloc[b * M1 + m1] = o;
                // the value after the last of the column before: to its CTA
                if (b == 0) {
                    if (c > 0) cluster.map_shared_rank(nbr, c - 1)[m1] = o.x;
                    else if (m1 > 0) cluster.map_shared_rank(nbr, kHeadCtas - 1)[m1 - 1] = o.x;
                }
            }
        }
    }
    if (P.bump_turn && c == 0 && tid == 0) *P.turn = turn + 1;
    if (!P.table) return;
    cluster.sync();  // the neighbours' values have landed
    for (int e = tid; e < Sh::per; e += nth) {
        const int b = e % Bc, m1 = e / Bc;
        const double2 o = vloc[b * M1 + m1];
        const double next = b + 1 < Bc ? vloc[(b + 1) * M1 + m1].x : nbr[m1];
        const int64_t m = 2 * (int64_t)(c * Bc + b + M2 * m1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t n = m + h;
            if (n >= P.n_out - 1) continue;
            const double a0 = h ? o.y : o.x, a1 = h ? next : o.y;
            if (!P.table_f32)
                reinterpret_cast<double2*>(P.table)[n] =
                    lik_entry0(a0, a1, P.bc[n], P.charge, P.inv_w);
            else
                reinterpret_cast<float2*>(P.table)[n] = make_float2(
                    (float)(P.charge * a0), (float)(P.charge * (a1 - a0) * P.inv_w));
        }
    }
}

// f(kernel, shape) for the plan's factors; false when there is no such kernel.
template <typename F>
bool for_shape(int M1, int M2, F f) {
    if (M1 == 64 && M2 == 64) f(head_fft_kernel<2, 2>, HeadShape<2, 2>{});
    else if (M1 == 64 && M2 == 128) f(head_fft_kernel<2, 4>, HeadShape<2, 4>{});
    else if (M1 == 128 && M2 == 128) f(head_fft_kernel<4, 4>, HeadShape<4, 4>{});
    else if (M1 == 128 && M2 == 256) f(head_fft_kernel<4, 8>, HeadShape<4, 8>{});
    else if (M1 == 256 && M2 == 256) f(head_fft_kernel<8, 8>, HeadShape<8, 8>{});
    else return false;
    return true;
}

}  // namespace

bool head_fft_takes(const SpecParams& P) {
    if (P.mode != (SPEC_FORWARD | SPEC_MULTIPLY | SPEC_INVERSE) || P.batch || P.general ||
        P.p.C != kHeadCtas || P.n_in > P.p.N || P.n_out > P.p.N)
        return false;
    bool fits = false;
    return for_shape(P.p.M1, P.p.M2,
                     [&](auto, auto sh) { fits = sh.bytes <= device_info().max_smem_optin &&
                                                 sh.L == P.p.L; }) &&
           fits;
}

// h_{d mod N} for |d| < S at position d mod M (the rest 0).
__global__ void extend_response_kernel(const double* y, int64_t N, int S, int64_t P, double* h) {
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < P;
         x += (int64_t)gridDim.x * blockDim.x)
        h[x] = x < S ? y[x] : (x > P - S ? y[N - (P - x)] : 0.0);
}

int64_t head_fft_length(int64_t N, int S) {
    if ((N & (N - 1)) == 0 || N < S) return 0;
    int64_t P = 8192;
    while (P < 2 * (int64_t)S - 1) P *= 2;
    SpecPlan plan;
    if (P > kMaxClusterFFT || !make_spec_plan(P, plan)) return 0;
    SpecParams q = {};
    q.p = plan;
    q.mode = SPEC_FORWARD | SPEC_MULTIPLY | SPEC_INVERSE;
    q.n_in = q.n_out = S;
    return head_fft_takes(q) ? P : 0;
}

int make_head_response(const double2* H, int64_t N, int S, int64_t P, double2** out) {
    *out = nullptr;
    double* y = nullptr;
    BB_CUDA(cudaMalloc((void**)&y, sizeof(double) * (size_t)(N + P)));
    int rc = blond_irfft_f64(reinterpret_cast<const double*>(H), N, y, N, nullptr);
    if (rc == BLOND_OK) {
        extend_response_kernel<<<64, 256>>>(y, N, S, P, y + N);
        if (cudaGetLastError() != cudaSuccess ||
            cudaMalloc((void**)out, sizeof(double2) * (size_t)(P / 2 + 1)) != cudaSuccess) {
            set_error("head: building the response failed");
            rc = BLOND_ERR_CUDA;
        }
    }
    if (rc == BLOND_OK)
        rc = blond_rfft_f64(y + N, P, P, reinterpret_cast<double*>(*out), nullptr);
    if (rc == BLOND_OK && cudaDeviceSynchronize() != cudaSuccess) {
        set_error("head: building the response failed");
        rc = BLOND_ERR_CUDA;
    }
    cudaFree(y);
    if (rc && *out) {
        cudaFree(*out);
        *out = nullptr;
    }
    return rc;
}

int prepare_head_fft() {
    static bool done[64] = {false};
    const DeviceInfo& d = device_info();
    if (done[d.device & 63]) return BLOND_OK;
    cudaError_t rc = cudaSuccess;
    const int shapes[5][2] = {{64, 64}, {64, 128}, {128, 128}, {128, 256}, {256, 256}};
    for (const auto& s : shapes)
        for_shape(s[0], s[1], [&](auto k, auto sh) {
            if (sh.bytes > d.max_smem_optin) return;
            if (rc == cudaSuccess)
                rc = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (rc == cudaSuccess)
                rc = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          sh.bytes);
        });
    BB_CUDA(rc);
    done[d.device & 63] = true;
    return BLOND_OK;
}

int launch_head_fft(const SpecParams& P, cudaStream_t stream) {
    int rc = prepare_head_fft();
    if (rc) return rc;
    cudaError_t ce = cudaSuccess;
    for_shape(P.p.M1, P.p.M2, [&](auto k, auto sh) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kHeadCtas);
        cfg.blockDim = dim3(kSpecThreads);
        cfg.dynamicSmemBytes = sh.bytes;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kHeadCtas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = P.pdl ? 2 : 1;
        ce = cudaLaunchKernelEx(&cfg, k, P);
    });
    BB_CUDA(ce);
    return BLOND_OK;
}

}  // namespace bb
