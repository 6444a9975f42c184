// tpsc_al.cu -- the Aslamazov-Larkin vertex correction chijj3(iq_n) of the
// current-current correlator, FP64 (cond_opt::calc_chijj_vertex_corr_all_optim
// with chi3 = true, src/cond_opt.cpp:4292-6420).
//
// The correction is evaluated on the reference's non-uniform bosonic grid
// (src/cond_opt.cpp:5123-5155); every grid frequency q_n runs the same
// pipeline on the K4 grid of interior kx points (c = l nbk + m,
// k = ((l+1), m) pi/(nbk-1), r folded into the octant):
//   once per call (launch_al_setup):
//    * G(r, tau_j) in FP64 (k_gslice); the branch's G(r, -tau) is
//      -G(r, beta - tau), its tau-derivatives at 0 and beta follow from the
//      hopping table and d/dtau G(r, 0+);
//    * hG slices: h(k, tau) -> DST x DCT -> times G(r, -tau) -> DST x DCT
//      (src/cond_opt.cpp:5158-5248), and their end slopes;
//    * per column pair: clamped spline of hG over tau, FFT -> hG(q, i q_p)
//      and its 1/q^2 coefficient (src/cond_opt.cpp:5250-5330);
//    * k_al_tables: chi0, hG, the RPA factors and the asymptote at every
//      frequency, the asymptote in tau and G(k, i k): what every grid
//      frequency reads;
//   per batch of grid frequencies (launch_al_freqs):
//    * k_al_hq: the difference quotient I_n(q, i q_m) of hG against chi0,
//      times the RPA vertices, minus its closed-form asymptote, FFT to tau,
//      plus the asymptote's closed form in tau (src/cond_opt.cpp:5351-5622);
//    * k_al_q2r: DST x DCT of Re and Im, q -> r (src/cond_opt.cpp:5628-5716);
//    * k_al_r2k: times G(r, -tau) for H(tau) and for the mirror
//      H2(tau) = H(beta - tau), DST x DCT back to k, and the four end slopes
//      (src/cond_opt.cpp:5718-5900, 5987-6180);
//    * k_al_tau: per k, the Re and Im splines of both, pre-twiddled FFTs to
//      fermionic frequencies, and the sum over k_m of
//      G(k, i k_m) G(k, i k_m + i q_n) (H - H2) (src/cond_opt.cpp:5906-5985,
//      6182-6398);
//    * k_al_finish: the per-k terms added in a fixed order, total and
//      angular bins.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tpsc_device.cuh"

namespace tpsc {

namespace {

// the AL branch's G(r, -tau_j) = DCT-I[G0(k, -tau_j)]/L^2 (src/cond_opt.cpp:4382-4410)
// from this library's G(r, tau): G(r, -tau) = -G(r, beta - tau), j = 0..Nw0
__device__ __forceinline__ double g_minus(const double *__restrict__ Grt, int nw0, int n8, int j, int o) {
    return -Grt[(size_t)(nw0 - j) * n8 + o];
}
// d/dtau G(r, -tau) at 0 (side 0) and beta (side 1) (src/cond_opt.cpp:4415-4446):
// DCT-I[(eps - mu0) n_F]/L^2 = er - mu0 delta_r0 - d/dtau G(r, 0+) at 0, and
// er - mu0 delta_r0 minus that at beta, i.e. d/dtau G(r, 0+)
__device__ __forceinline__ double dg_minus(const double *__restrict__ er, const double *__restrict__ dG0p, double mu0,
                                           int side, int o) {
    return side == 0 ? ((o == 0 ? -mu0 : er[o]) - dG0p[o]) : dG0p[o];
}

// complex helpers on double2
__device__ __forceinline__ double2 cneg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ double2 cmuli(double2 a) { return make_double2(-a.y, a.x); }  // i a
__device__ __forceinline__ double2 crs(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
__device__ __forceinline__ double2 cinv(double2 b) { return cdiv(make_double2(1.0, 0.0), b); }

// exp(-i pi m / N) for any m >= 0, from the table ht[m] = exp(+i pi m / N), m < N
__device__ __forceinline__ double2 half_twiddle_conj(const TwoLevelTw *ht2, int m, int N) {
    m %= 2 * N;
    const double2 h = tw_at(ht2, m < N ? m : m - N);
    return m < N ? make_double2(h.x, -h.y) : make_double2(-h.x, h.y);
}

// ---------------------------------------------------------------------------
// once per call
// ---------------------------------------------------------------------------

// h G(q, tau_j), j = blockIdx.x = 0..Nw0: h(k, tau_j) from the (eps - mu0, A)
// table (src/cond_opt.cpp:4304-4330), DST x DCT, times G(r, -tau_j), DST x DCT
// (src/cond_opt.cpp:5220-5248); h(r, 0) and h(r, beta) kept for the end slopes.
template <int NBK>
__global__ void __launch_bounds__(SlicePlan<NBK>::threads, SlicePlan<NBK>::blocks)
    k_al_hg_slice(const double *__restrict__ tab, const double *__restrict__ Grt, const double2 *__restrict__ tw,
                  int nw0, int n8, double T, double *__restrict__ hGt, double *__restrict__ pre) {
    constexpr int K4 = (NBK - 2) * NBK;
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK>(S, tw);
    const int j = blockIdx.x;
    const double t = j / (nw0 * T);
    const double bt = 1.0 / T - t;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const double2 xa = *reinterpret_cast<const double2 *>(tab + 4 * c);
        S[c] = xa.y * exp(xa.x > 0 ? -xa.x * t : xa.x * bt);
    }
    __syncthreads();
    plan_dst_dct<NBK>(S, tws);
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const int l = c / NBK, m = c % NBK;
        const double v = S[c];
        if (j == 0) pre[c] = v;
        if (j == nw0) pre[K4 + c] = v;
        S[c] = v * g_minus(Grt, nw0, n8, j, oct_index(l + 1, m));
    }
    __syncthreads();
    plan_dst_dct<NBK>(S, tws);
    for (int c = threadIdx.x; c < K4; c += blockDim.x) hGt[bidx2(j, c, nw0 + 1)] = S[c];
}

// End slopes of h G over tau (src/cond_opt.cpp:5158-5216): kind 0 (tau = 0),
// 1 (tau = beta): DST x DCT[ dh(r) G(r, -tau) + h(r) d/dtau G(r, -tau) ], with
// dh the transformed tau-derivative of h at that end (src/cond_opt.cpp:2744-2783).
template <int NBK>
__global__ void __launch_bounds__(kSliceThreads, 1)
    k_al_hg_bound(const double *__restrict__ ek, const double *__restrict__ dek, const double *__restrict__ er,
                  const double *__restrict__ dG0p, const double *__restrict__ Grt, const double2 *__restrict__ tw,
                  const double *__restrict__ pre, int nw0, int n8, double mu0, double T, double nf,
                  double *__restrict__ dhG) {
    constexpr int K4 = (NBK - 2) * NBK;
    extern __shared__ __align__(16) double S[];
    const auto *tws = slice_twiddles<NBK, SliceGroups<NBK>::wide>(S, tw);
    const int kind = blockIdx.x;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const int l = c / NBK, m = c % NBK;
        const double x = ek[oct_index(l + 1, m)] - mu0;
        const double d = nf * dek[c];
        double v;
        if (x > 0) {
            const double ep = exp(-x / T), q = ep + 1.0;
            v = kind == 0 ? -d * x / q : -d * x * ep / q;
        } else {
            const double en = exp(x / T), q = en + 1.0;
            v = kind == 0 ? -d * x * en / q : -d * x / q;
        }
        S[c] = v;
    }
    __syncthreads();
    dst_dct_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    const int jend = kind == 0 ? 0 : nw0;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const int l = c / NBK, m = c % NBK;
        const int o = oct_index(l + 1, m);
        S[c] = S[c] * g_minus(Grt, nw0, n8, jend, o) + pre[kind * K4 + c] * dg_minus(er, dG0p, mu0, kind, o);
    }
    __syncthreads();
    dst_dct_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    for (int c = threadIdx.x; c < K4; c += blockDim.x) dhG[kind * K4 + c] = S[c];
}

// shared memory of the per-pair tau kernel: two staged columns, one FFT
// buffer, the two-level twiddle tables
template <int N>
struct AlHgTauSmem {
    static constexpr size_t r_bytes = ((size_t)2 * (N + 1) * sizeof(double) + 15) & ~(size_t)15;
    static constexpr size_t tables_off = r_bytes + (size_t)padded_len(N) * sizeof(double2);
    static constexpr size_t bytes = tables_off + 2 * sizeof(TwoLevelTw);
};

// h G(q, i q_p) from h G(q, tau), one column pair per CTA (src/cond_opt.cpp:5250-5330):
// clamped spline with the end slopes, F_p = sum_j 6 a_j exp(-2 pi i jp/N);
// p = 0: 2 x the spline's integral; 0 < p < N/2: 2 Re[(1 - exp(-2 pi i p/N)) F_p];
// then hg2 = 2 (dhG(0) - dhG(beta)), the coefficient of -1/q^2.
template <int N>
__global__ void __launch_bounds__(256, 1)
    k_al_hg_tau(const double *__restrict__ hGt, const double *__restrict__ dhG, const double *__restrict__ spl,
                const double2 *__restrict__ tw, const double2 *__restrict__ ht, double T, int K4,
                double *__restrict__ hgq) {
    constexpr int NJ = N + 1, NO = N / 2, G = FftPlan<N>::G;
    extern __shared__ __align__(16) double R[];
    double2 *X = reinterpret_cast<double2 *>(reinterpret_cast<char *>(R) + AlHgTauSmem<N>::r_bytes);
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(R) + AlHgTauSmem<N>::tables_off);
    __shared__ double d0s[2], dNs[2], sV[2], sM[2], V0[2], VN[2];
    const int tid = threadIdx.x;
    tau_tables(tw2, tw2 + 1, tw, ht, N);
    const int c0 = 2 * blockIdx.x;
    stage_pair(R, hGt + (size_t)blockIdx.x * 2 * NJ, NJ, c0 + 1 < K4);
    if (tid < 2) {
        const int c = c0 + tid;
        d0s[tid] = c < K4 ? dhG[c] : 0.0;
        dNs[tid] = c < K4 ? dhG[K4 + c] : 0.0;
    }
    __syncthreads();
    if (tid < 2) {
        V0[tid] = R[tid * NJ];
        VN[tid] = R[tid * NJ + N];
    }
    column_sums<2>(R, NJ, 0, NJ, sV);
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_second_derivatives<2>(R, NJ, NJ, h, d0s, dNs, spl, spl + NJ);
    column_sums<2>(R, NJ, 0, NJ, sM);
    if (tid < G) {
        const double *Ma = R, *Mb = R + NJ;
        auto in = [&](int j) -> double2 { return make_double2((Ma[j + 1] - Ma[j]) * ih, (Mb[j + 1] - Mb[j]) * ih); };
        group_fft_io<N, -1>(X, tid, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
    }
    __syncthreads();
    for (int p = tid; p < NO; p += blockDim.x) {
        double2 F[2];
        if (p > 0) split_real(X[pidx(p)], X[pidx(N - p)], F[0], F[1]);
        const double2 w = tw_at(tw2, p);
        const double2 f = make_double2(1.0 - w.x, -w.y);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int c = c0 + q;
            if (c >= K4) continue;
            double v;
            if (p == 0) {
                const double M0 = R[q * NJ], MN = R[q * NJ + N];
                v = 2.0 * (h * (sV[q] - 0.5 * (V0[q] + VN[q])) - h * h * h / 24.0 * (2.0 * sM[q] - M0 - MN));
            } else {
                v = 2.0 * (f.x * F[q].x - f.y * F[q].y);
            }
            hgq[(size_t)c * (NO + 1) + p] = v;
        }
    }
    if (tid < 2 && c0 + tid < K4) hgq[(size_t)(c0 + tid) * (NO + 1) + NO] = 2.0 * (d0s[tid] - dNs[tid]);
}

// ---------------------------------------------------------------------------
// what the grid frequencies share, once per call
// ---------------------------------------------------------------------------
struct AlTabArgs {
    const double *chiq;            // chi0(q, i q_p), p <= NO, column blocks
    const double *cinf, *cinf2;    // [n8] its 1/q^2, 1/q^4 tail coefficients
    const double *hgq;             // [K4 (NO+1)]
    const double2 *S;              // Sigma as in AlTauArgs
    const double *s2, *s3, *sinf, *ek;
    double4 *tab;                  // [K4 (N+1)] (chi0, hG, RPA factor, asymptote) at q_p, p = 0..N
    double *shape;                 // two-column blocks: the asymptote's closed form at tau_j
    double2 *dshape;               // [2 K4] its tau-derivatives at 0 and beta
    double2 *gk;                   // [K4 N] G(k, i k_f), f = 0..N-1
    int K4, nbk, N;
    double T, mu, Usp, Uch;
};

// One column c per CTA.  chi0 and hG beyond the stored frequencies by their
// tails; the RPA factor 3 Usp chisp + Uch chich and the asymptote Hinf(q_p) of
// the difference quotient's product, Hinf(tau_j) in closed form with its end
// slopes (src/cond_opt.cpp:5351-5622), and G(k, i k_f)
// (src/cond_opt.cpp:6253-6290).  They do not depend on the grid frequency: per
// frequency they cost k_al_hq and k_al_tau 15 divisions, two complex
// exponentials, two exponentials and two Sigma reads per point.
__global__ void __launch_bounds__(128) k_al_tables(const AlTabArgs a) {
    const int c = blockIdx.x, l = c / a.nbk, m = c % a.nbk, o = oct_index(l + 1, m);
    const int N = a.N, NO = N / 2, NB = NO + 1, NJ = N + 1;
    const double T = a.T, Usp = a.Usp, Uch = a.Uch, tp = 2.0 * kPi * T;
    const double *hq = a.hgq + (size_t)c * (NO + 1);
    const double ci = a.cinf[o], ci2 = a.cinf2[o], hg2 = hq[NO];
    for (int p = threadIdx.x; p <= N; p += blockDim.x) {
        const double wn = tp * p, w2 = wn * wn;
        const double ch = p <= NO ? a.chiq[bidx(p, o, NB)] : ci / w2 + ci2 / (w2 * w2);
        const double hg = p == 0 ? hq[0] : -hg2 / w2 + hq[p < NO ? p : NO - 1] / (w2 * w2);
        const double pre = 3 * Usp * (ch / (1.0 - Usp * ch / 2)) + Uch * (ch / (1.0 + Uch * ch / 2));
        const double hinf =
            hg2 * (3.0 * Usp * (1.0 / (-w2 + Usp * ci / 2.0)) + Uch * (1.0 / (-w2 - Uch * ci / 2.0)));
        a.tab[(size_t)c * NJ + p] = make_double4(ch, hg, pre, hinf);
    }
    // spin poles +-i sqrt(Usp ci/2), charge poles +-sqrt(Uch ci/2)
    const double zs = sqrt(Usp * ci / 2.0), zch0 = sqrt(Uch * ci / 2.0), zch1 = -zch0;
    const double2 zsp0 = make_double2(0.0, zs), zsp1 = make_double2(-0.0, -zs);
    const double2 one = make_double2(1.0, 0.0);
    const double2 dsp0 = cmul(csub(cexp2(cscale(zsp0, -1.0 / T)), one), csub(zsp0, zsp1));
    const double2 dsp1 = cmul(csub(cexp2(cscale(zsp1, -1.0 / T)), one), csub(zsp1, zsp0));
    const double dch0 = (exp(-zch0 / T) - 1.0) * (zch0 - zch1), dch1 = (1.0 - exp(zch1 / T)) * (zch1 - zch0);
    for (int j = threadIdx.x; j <= N; j += blockDim.x) {
        const double t = j / (N * T);
        // (the two spin poles are conjugate: their sum is real)
        const double tsp = cadd(cdiv(cexp2(cscale(zsp0, -t)), dsp0), cdiv(cexp2(cscale(zsp1, -t)), dsp1)).x;
        const double tch = exp(-zch0 * t) / dch0 + exp(zch1 * (1.0 / T - t)) / dch1;
        a.shape[bidx2(j, c, NJ)] = hg2 * (3.0 * Usp * tsp + Uch * tch);
    }
    if (threadIdx.x < 2) {
        const int side = threadIdx.x;
        const double2 e0 = side ? cexp2(cscale(zsp0, -1.0 / T)) : one, e1 = side ? cexp2(cscale(zsp1, -1.0 / T)) : one;
        const double2 tsp = csub(cneg(cdiv(cmul(zsp0, e0), dsp0)), cdiv(cmul(zsp1, e1), dsp1));
        const double tch = side ? -zch0 * exp(-zch0 / T) / dch0 - zch1 / dch1
                                : -zch0 / dch0 - zch1 * exp(zch1 / T) / dch1;
        a.dshape[(size_t)side * a.K4 + c] = crs(hg2, cadd(crs(3.0 * Usp, tsp), make_double2(Uch * tch, 0.0)));
    }
    const double e = a.ek[o], sinf = a.sinf[0], C2 = a.s2[o], C3 = a.s3[o];
    for (int f = threadIdx.x; f < N; f += blockDim.x) {
        const double kn = (2 * f + 1) * kPi * T;
        double sr = -C2 / (kn * kn), si = -sinf / kn + C3 / (kn * kn * kn);
        if (f < NO) {
            const double2 Sv = a.S[bidx(f, o, NO)];
            const double k4 = kn * kn * kn * kn;
            sr += Sv.x / k4;
            si += Sv.y / k4;
        }
        a.gk[(size_t)c * N + f] = cinv(make_double2(-e + a.mu - sr, kn - si));
    }
}

// ---------------------------------------------------------------------------
// per grid frequency q_nn; blockIdx.y (blockIdx.x of the slices' planes) is the
// frequency's place in the launch's batch
// ---------------------------------------------------------------------------
struct AlHqArgs {
    const double4 *tab;
    const double *shape;
    const double2 *dshape;
    const double2 *tw, *ht;        // [N] FFT twiddles, half-step twiddles
    const int *ind;                // the batch's frequencies
    double2 *HQ, *dHQ;
    int K4, K4p;
    double T;
};

// threads of a column pair's CTA: one FFT group
template <int N>
struct AlHqPlan {
    static constexpr int G = FftPlan<N>::G;
    static constexpr int threads = G < 32 ? 32 : G;
    static constexpr size_t smem = (size_t)padded_len(N) * sizeof(double2) + 2 * sizeof(TwoLevelTw);
};

// I_n(q, i q_m) -> H(q, tau) for one column pair per CTA (src/cond_opt.cpp:5351-5622):
//   m in [0, NO - nc): p1 = m, p2 = m + nn; m in [NO - nc, N): p1 = m - N, p2 = p1 + nn;
//   I = (3 Usp chisp(p1) + Uch chich(p1)) (hG(p1) - hG(p2)) / (chi0(p1) - chi0(p2)),
//   with (4 D(m-1) - D(m-2))/3 for the quotient D where p1 = p2 (nn even);
//   ft_m = T (I - Hinf(q_m)), H(q, tau_j) = FFT_{-}[ft]_j + Hinf(tau_j), closed form.
// Bound: the FP64 pipe (one division and the FFT per point) and the FFT's
// exchange.  One FFT group per CTA, so that no thread idles in the transform
// and six CTAs share an SM; 64^2 x 1024: 150 -> 15 us a frequency against 256
// threads of which 64 transform and every asymptote formed anew.
template <int N>
__global__ void __launch_bounds__(AlHqPlan<N>::threads) k_al_hq(const AlHqArgs a) {
    constexpr int NO = N / 2, G = FftPlan<N>::G, NJ = N + 1, NT = AlHqPlan<N>::threads;
    extern __shared__ __align__(16) double2 X[];
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(X + padded_len(N));
    __shared__ double sums[2];
    const int tid = threadIdx.x;
    const int c0 = 2 * blockIdx.x, nn = a.ind[blockIdx.y], nc = nn / 2;
    const double T = a.T, tp = 2.0 * kPi * T;
    tau_tables(tw2, tw2 + 1, a.tw, a.ht, N);  // published by block_sum's barrier
    const double4 *tab[2] = {a.tab + (size_t)c0 * NJ, a.tab + (size_t)min(c0 + 1, a.K4 - 1) * NJ};
    auto quot = [&](const double4 *t, int p1, int p2) -> double {
        const double4 u = t[abs(p1)], v = t[abs(p2)];
        return (u.y - v.y) / (u.x - v.x);
    };
    // ---- the quotient minus its asymptote, packed as Re/Im of one FFT
    double acc[2] = {0.0, 0.0};
    for (int m = tid; m < N; m += NT) {
        const bool first = m < NO - nc;
        const int p1 = first ? m : m - N, p2 = p1 + nn;
        const double wn = tp * p1;
        double ft[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double4 u = tab[k][abs(p1)], v = tab[k][abs(p2)];
            double D = (u.y - v.y) / (u.x - v.x);
            if (!first && (nn % 2) == 0 && m - N == -(nn / 2))
                D = (4 * quot(tab[k], p1 - 1, p2 - 1) - quot(tab[k], p1 - 2, p2 - 2)) / 3.0;
            ft[k] = T * (u.z * D - u.w);
            acc[k] += wn * ft[k];
        }
        X[pidx(m)] = make_double2(ft[0], ft[1]);
    }
    block_sum<2>(acc, sums);
    if (tid < G) group_fft<N, -1>(X, tid, (const TwoLevelTw *)tw2, 0);
    __syncthreads();
    // ---- back in tau: the FFT part plus the asymptote's closed form
    double2 *HQ = a.HQ + (size_t)blockIdx.y * NJ * a.K4p;
    const double2 *shape = reinterpret_cast<const double2 *>(a.shape) + (size_t)blockIdx.x * NJ;
    const bool two = c0 + 1 < a.K4;
    for (int j = tid; j <= N; j += NT) {
        const int k = j & (N - 1);
        double2 F[2];
        split_real(X[pidx(k)], X[pidx((N - k) & (N - 1))], F[0], F[1]);
        const double2 hinf = shape[j];
        double2 *dst = HQ + (size_t)j * a.K4p + c0;
        dst[0] = make_double2(F[0].x + hinf.x, F[0].y);
        if (two) dst[1] = make_double2(F[1].x + hinf.y, F[1].y);
    }
    // the end slopes: i dt0 (src/cond_opt.cpp:5539-5546) plus the asymptote's
    if (tid < 4 && c0 + (tid & 1) < a.K4) {
        const int q = tid & 1, side = tid >> 1, c = c0 + q;
        a.dHQ[((size_t)blockIdx.y * 2 + side) * a.K4 + c] =
            cadd(make_double2(0.0, -sums[q]), a.dshape[(size_t)side * a.K4 + c]);
    }
}

// The slice kernels of H: up to 65 lines the slice is complex in shared memory, one
// transform a line (the lines' real and imaginary parts are what two real lines are to
// the packed transforms elsewhere), so that H is read and written whole: as two real
// slices one after the other every 16-byte value took two half-used accesses, and L1
// was the busiest unit (68%).  129 lines do not fit and keep the two real slices.
// Per launch of 10 frequencies at 64^2 x 1024: r -> k 437 -> 338 us, q -> r 140 -> 133;
// 32^2 x 256: 100 -> 58 and 41 -> 26; 128^2 x 256: 179 -> 142 and 59 -> 50.
template <int NBK>
struct AlSlice {
    static constexpr bool cplx = NBK <= 65;
    static constexpr int L = 2 * (NBK - 1), G = FftPlan<L>::G;
    using F = SymFft<L >= 64 ? L : 64>;
    static constexpr bool sym = NBK >= 33;  // as SlicePlan: below, symmetry saves nothing
    static constexpr int warps = NBK == 65 ? 5 : NBK == 33 ? 4 : 2;
    static constexpr int threads = cplx ? 32 * warps : SlicePlan<NBK>::threads;
    static constexpr int blocks = !cplx ? SlicePlan<NBK>::blocks : NBK == 65 ? 2 : NBK == 33 ? 4 : 8;
    static constexpr size_t scr_off = (size_t)(NBK - 2) * NBK * sizeof(double2);
    static constexpr size_t scr = (size_t)(sym ? warps * F::per_warp * F::len : threads / G * padded_len(L)) * sizeof(double2);
    static constexpr size_t tw_off = scr_off + scr;
    static constexpr size_t bytes = cplx ? tw_off + (sym ? F::ntw : L) * sizeof(double2) : SlicePlan<NBK>::bytes;
    static_assert(bytes + 1024 <= 233472 / blocks || !cplx, "the CTAs of an SM share its memory");
};
template <int NBK>
__device__ __forceinline__ void al_twiddles(double2 *S, const double2 *__restrict__ tw) {
    using P = AlSlice<NBK>;
    double2 *t = reinterpret_cast<double2 *>(reinterpret_cast<char *>(S) + P::tw_off);
    if constexpr (P::sym)
        for (int i = threadIdx.x; i < P::F::ntw; i += blockDim.x) t[i] = __ldg(&tw[(i / P::F::G + 1) * (i % P::F::G)]);
    else
        for (int i = threadIdx.x; i < P::L; i += blockDim.x) t[i] = __ldg(&tw[i]);
}
// DST-I along l (NBK - 2) x DCT-I along m (NBK) of the complex slice S, in place;
// ends with a barrier
template <int NBK>
__device__ __forceinline__ void al_dst_dct(double2 *S) {
    using P = AlSlice<NBK>;
    constexpr int L = P::L, NR = NBK - 2;
    double2 *scr = reinterpret_cast<double2 *>(reinterpret_cast<char *>(S) + P::scr_off);
    const double2 *tw = reinterpret_cast<const double2 *>(reinterpret_cast<char *>(S) + P::tw_off);
    auto row_in = [&](int p, int j) -> double2 { return S[p * NBK + (j < NBK ? j : L - j)]; };
    auto row_out = [&](int p, int k, double2 z) { S[p * NBK + k] = z; };
    // z = [0, X, 0, -reverse(X)]: its transform is -i Y
    auto col_in = [&](int p, int j) -> double2 {
        if (j == 0 || j == NR + 1) return make_double2(0.0, 0.0);
        const double2 x = S[(j <= NR ? j - 1 : L - j - 1) * NBK + p];
        return j <= NR ? x : make_double2(-x.x, -x.y);
    };
    auto col_out = [&](int p, int k, double2 z) {
        if (k >= 1 && k <= NR) S[(k - 1) * NBK + p] = make_double2(-z.y, z.x);
    };
    if constexpr (P::sym) {
        sym_lines<L, 1>(scr, tw, NR, row_in, row_out);
        __syncthreads();
        sym_lines<L, -1>(scr, tw, NBK, col_in, col_out);
        __syncthreads();
    } else {
        constexpr int G = P::G;
        const int grp = threadIdx.x / G, t = threadIdx.x % G, ngrp = blockDim.x / G;
        double2 *x = scr + grp * padded_len(L);
#pragma unroll 1
        for (int p = grp; p < NR; p += ngrp) {
            group_fft_io<L, -1, true>(
                x, t, tw, grp, [&](int j) { return row_in(p, j); },
                [&](int k, double2 z) {
                    if (k < NBK) row_out(p, k, z);
                });
            if constexpr (FftPlan<L>::NPASS == 1) group_sync<G>(grp);
        }
        __syncthreads();
#pragma unroll 1
        for (int p = grp; p < NBK; p += ngrp) {
            group_fft_io<L, -1, true>(
                x, t, tw, grp, [&](int j) { return col_in(p, j); }, [&](int k, double2 z) { col_out(p, k, z); });
            if constexpr (FftPlan<L>::NPASS == 1) group_sync<G>(grp);
        }
        __syncthreads();
    }
}

// H(q, tau_j) -> H(r, tau_j) = DST x DCT[nf H] of the real and imaginary parts
// (src/cond_opt.cpp:5628-5716); blocks Nw0 + 1 and Nw0 + 2 transform the two
// end slopes.
template <int NBK>
__global__ void __launch_bounds__(AlSlice<NBK>::threads, AlSlice<NBK>::blocks)
    k_al_q2r(const double2 *__restrict__ HQ, const double2 *__restrict__ dHQ, const double2 *__restrict__ tw,
             int nw0, double nf, double2 *__restrict__ HR, double2 *__restrict__ dHR) {
    constexpr int K4 = (NBK - 2) * NBK, K4p = (K4 + 1) & ~1;
    extern __shared__ __align__(16) double S[];
    const int b = blockIdx.x, NJ = nw0 + 1;
    const size_t row = (size_t)blockIdx.y * NJ + b, drow = (size_t)blockIdx.y * 2 + (b - NJ);
    const double2 *src = b < NJ ? HQ + row * K4p : dHQ + drow * K4;
    double2 *dst2 = b < NJ ? HR + row * K4p : dHR + drow * K4;
    if constexpr (AlSlice<NBK>::cplx) {
        double2 *Z = reinterpret_cast<double2 *>(S);
        al_twiddles<NBK>(Z, tw);
        batched<4>(K4, [&](int c) { return src[c]; }, [&](int c, double2 v) { Z[c] = cscale(v, nf); });
        __syncthreads();
        al_dst_dct<NBK>(Z);
        for (int c = threadIdx.x; c < K4; c += blockDim.x) dst2[c] = Z[c];
        return;
    }
    const auto *tws = plan_twiddles<NBK>(S, tw);
    double *dst = reinterpret_cast<double *>(dst2);
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        for (int c = threadIdx.x; c < K4; c += blockDim.x) S[c] = nf * (part == 0 ? src[c].x : src[c].y);
        __syncthreads();
        plan_dst_dct<NBK>(S, tws);
        for (int c = threadIdx.x; c < K4; c += blockDim.x) dst[2 * c + part] = S[c];
        __syncthreads();
    }
}

// H(r, tau_j) G(r, -tau_j) and H2(r, tau_j) G(r, -tau_j), H2(r, tau) = H(r, beta - tau),
// -> DST x DCT to k, real and imaginary parts (src/cond_opt.cpp:5845-5900, 6125-6180),
// into the two-column-block layouts of HK and H2K.  Blocks Nw0 + 1 + k, k < 4,
// transform the end slopes (src/cond_opt.cpp:5729-5843, 6004-6123):
//   k = 0: H(r, 0) dG(0) + dH(r, 0) G(r, 0);   k = 1: H(r, beta) dG(beta) + dH(r, beta) G(r, -beta);
//   k = 2, 3: the same for H2, whose end values are H(r, beta), H(r, 0) and
//   whose end slopes are -dH(r, beta), -dH(r, 0).
template <int NBK>
__global__ void __launch_bounds__(AlSlice<NBK>::threads, AlSlice<NBK>::blocks)
    k_al_r2k(const double2 *__restrict__ HR, const double2 *__restrict__ dHR, const double *__restrict__ Grt,
             const double *__restrict__ er, const double *__restrict__ dG0p, const double2 *__restrict__ tw, int nw0,
             int n8, double mu0, double2 *__restrict__ HK, double2 *__restrict__ H2K, double2 *__restrict__ dHK) {
    constexpr int K4 = (NBK - 2) * NBK, K4p = (K4 + 1) & ~1;
    extern __shared__ __align__(16) double S[];
    const int b = blockIdx.x, NJ = nw0 + 1;
    HR += (size_t)blockIdx.y * NJ * K4p;
    dHR += (size_t)blockIdx.y * 2 * K4;
    HK += (size_t)blockIdx.y * NJ * K4p;
    H2K += (size_t)blockIdx.y * NJ * K4p;
    dHK += (size_t)blockIdx.y * 4 * K4;
    if constexpr (AlSlice<NBK>::cplx) {
        double2 *Z = reinterpret_cast<double2 *>(S);
        al_twiddles<NBK>(Z, tw);
        const int nh = b < NJ ? 2 : 1;
#pragma unroll 1
        for (int h = 0; h < nh; ++h) {
            auto put = [&](int c, double2 v) { Z[c] = v; };
            if (b < NJ) {
                const double2 *hr = HR + (size_t)(h == 0 ? b : nw0 - b) * K4p;
                batched<4>(
                    K4,
                    [&](int c) {
                        const int l = c / NBK, m = c % NBK;
                        return cscale(hr[c], g_minus(Grt, nw0, n8, b, oct_index(l + 1, m)));
                    },
                    put);
            } else {
                const int k = b - NJ, side = k & 1;  // 0: tau = 0, 1: beta
                const double2 *hr = HR + (size_t)((k == 0 || k == 3) ? 0 : nw0) * K4p;      // H at 0 / beta
                const double2 *dr = dHR + (size_t)((k == 0 || k == 3) ? 0 : 1) * K4;        // which dH
                const double sg = k < 2 ? 1.0 : -1.0;
                for (int c = threadIdx.x; c < K4; c += blockDim.x) {
                    const int o = oct_index(c / NBK + 1, c % NBK);
                    put(c, cadd(cscale(hr[c], dg_minus(er, dG0p, mu0, side, o)),
                                cscale(dr[c], sg * g_minus(Grt, nw0, n8, side == 0 ? 0 : nw0, o))));
                }
            }
            __syncthreads();
            al_dst_dct<NBK>(Z);
            double2 *dst = h == 0 ? HK : H2K;
            for (int c = threadIdx.x; c < K4; c += blockDim.x) {
                if (b < NJ)
                    dst[bidx2(b, c, NJ)] = Z[c];
                else
                    dHK[(size_t)(b - NJ) * K4 + c] = Z[c];
            }
            __syncthreads();
        }
        return;
    }
    const auto *tws = plan_twiddles<NBK>(S, tw);
    const int npass = b < NJ ? 4 : 2;
#pragma unroll 1
    for (int pass = 0; pass < npass; ++pass) {
        const int part = pass & 1;
        for (int c = threadIdx.x; c < K4; c += blockDim.x) {
            const int l = c / NBK, m = c % NBK;
            const int o = oct_index(l + 1, m);
            const double *hr = reinterpret_cast<const double *>(HR);
            const double *dr = reinterpret_cast<const double *>(dHR);
            double v;
            if (b < NJ) {
                const int row = pass < 2 ? b : nw0 - b;
                v = hr[2 * ((size_t)row * K4p + c) + part] * g_minus(Grt, nw0, n8, b, o);
            } else {
                const int k = b - NJ;
                const int side = k & 1;                                        // 0: tau = 0, 1: beta
                const int row = (k == 0 || k == 3) ? 0 : nw0;                  // H at 0 / beta
                const int sl = (k == 0) ? 0 : (k == 1) ? 1 : (k == 2) ? 1 : 0;  // which dH
                const double sg = k < 2 ? 1.0 : -1.0;
                v = hr[2 * ((size_t)row * K4p + c) + part] * dg_minus(er, dG0p, mu0, side, o) +
                    sg * dr[2 * ((size_t)sl * K4 + c) + part] * g_minus(Grt, nw0, n8, side == 0 ? 0 : nw0, o);
            }
            S[c] = v;
        }
        __syncthreads();
        plan_dst_dct<NBK>(S, tws);
        for (int c = threadIdx.x; c < K4; c += blockDim.x) {
            double *dst;
            if (b < NJ)
                dst = reinterpret_cast<double *>((pass < 2 ? HK : H2K) + bidx2(b, c, NJ));
            else
                dst = reinterpret_cast<double *>(dHK + (size_t)(b - NJ) * K4 + c);
            dst[part] = S[c];
        }
        __syncthreads();
    }
}

struct AlTauArgs {
    const double2 *HK, *H2K, *dHK;
    const double2 *gk;   // [K4 N] G(k, i k_f)
    const double *dek;
    const double *spl;
    const double2 *tw, *ht;
    const int *ind;
    double *colv;
    int K4, K4p, nbk;
    double T, U, nf;
};

// shared memory of k_al_tau: the complex columns of H and H2, each splined and
// transformed in place, and the twiddle tables
template <int N>
struct AlTauPlan {
    static constexpr int G = FftPlan<N>::G;
    static constexpr int threads = 2 * G < 32 ? 32 : 2 * G;
    static constexpr int x_len = padded_len(N) + 2;  // N + 1 nodes
    static constexpr size_t smem = (size_t)2 * x_len * sizeof(double2) + 2 * sizeof(TwoLevelTw);
};

// One k point per CTA, a group of G threads for each of H and H2: the splines of
// the real and imaginary parts over tau with their end slopes,
// F_j = sum_l exp(-i pi l/N) 6 (a_l^Re + i a_l^Im) exp(-2 pi i lj/N)
// (src/cond_opt.cpp:5906-5985, 6187-6251), the fermionic values
//   H(i w) = -i C1/w - C2/w^2 + i C3/w^3 + (1 - exp(-i (2f+1) pi/N)) F/w^4
// (H at k_m + q_nn, H2 at k_m), and the term
//   -i U T nf wt dek sum_m G(k, i k_m) G(k, i k_m + i q_nn) (H - H2) / (2 q_nn)
// (src/cond_opt.cpp:6253-6398); its real part -> colv[c].
// Bound: the dependent spline sweeps and the FFTs' exchange.  Both transforms
// run at once, each in place in its column's buffer (35 KB a CTA at N = 1024
// instead of 53), so that four CTAs of busy threads share an SM; 64^2 x 1024:
// 167 -> 46 us a frequency (one after the other in 256 threads, 64 of them in
// the FFT, with G(k, i k) formed at every point).
template <int N>
__global__ void __launch_bounds__(AlTauPlan<N>::threads, AlTauPlan<N>::threads <= 128 ? 4 : 1)
    k_al_tau(const AlTauArgs a) {
    constexpr int NO = N / 2, G = FftPlan<N>::G, NJ = N + 1, NT = AlTauPlan<N>::threads;
    extern __shared__ __align__(16) double2 X1[];
    double2 *X2 = X1 + AlTauPlan<N>::x_len;
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(X2 + AlTauPlan<N>::x_len);
    const TwoLevelTw *ht2 = tw2 + 1;
    __shared__ double2 cw[2], dsum[2], d2sum[2];
    __shared__ double sums[1];
    const int tid = threadIdx.x;
    const int c = blockIdx.x, nn = a.ind[blockIdx.y], nc = nn / 2;
    const double T = a.T, h = 1.0 / (N * T), ih = 1.0 / h, pT = kPi * T;
    tau_tables(tw2, tw2 + 1, a.tw, a.ht, N);
    const size_t plane = (size_t)blockIdx.y * NJ * a.K4p;
    for (int j = tid; j < NJ; j += NT) {
        X1[pidx(j)] = a.HK[plane + bidx2(j, c, NJ)];
        X2[pidx(j)] = a.H2K[plane + bidx2(j, c, NJ)];
    }
    __syncthreads();
    const int which = tid / G;
    if (which < 2) {
        const int t = tid % G;
        double2 *X = which == 0 ? X1 : X2;
        const double2 *dh = a.dHK + ((size_t)blockIdx.y * 4 + 2 * which) * a.K4 + c;
        const double2 d0 = dh[0], dN = dh[a.K4];
        if (t == 0) {
            cw[which] = cadd(X[0], X[pidx(N)]);
            dsum[which] = cadd(d0, dN);
        }
        group_sync<G>(which);
        spline_complex<N>(X, NJ, t, which, h, d0, dN, a.spl, a.spl + NJ);
        if (t == 0) d2sum[which] = cadd(X[0], X[pidx(N)]);
        auto in = [&](int j) -> double2 {
            const double2 e = tw_at(ht2, j);
            const double2 u = X[pidx(j)], v = X[pidx(j + 1)];
            return cmul(make_double2(e.x, -e.y), make_double2((v.x - u.x) * ih, (v.y - u.y) * ih));
        };
        group_fft_io<N, -1, false, true>(X, t, (const TwoLevelTw *)tw2, which, in, ScratchIO{X});
    }
    __syncthreads();
    // ---- the sum over k_m
    const double2 *gk = a.gk + (size_t)c * N;
    auto green = [&](int f) -> double2 {
        const double2 g = gk[f >= 0 ? f : -f - 1];
        return f >= 0 ? g : cconj(g);
    };
    auto hval = [&](double2 cwv, double2 ds, double2 d2s, double w, bool has, double2 Fv, int ph) -> double2 {
        const double i1 = 1.0 / w, i2 = i1 * i1, i3 = i2 * i1, i4 = i2 * i2;
        double2 v = cadd(csub(cmuli(cscale(cwv, -i1)), cscale(ds, i2)), cmuli(cscale(d2s, i3)));
        if (has) {
            const double2 ex = half_twiddle_conj(ht2, ph, N);
            v = cadd(v, cscale(cmul(make_double2(1.0 - ex.x, -ex.y), Fv), i4));
        }
        return v;
    };
    double acc[1] = {0.0};
    for (int j = tid; j < N; j += NT) {
        const bool first = j < NO - nc;
        const int f1 = first ? j : j - N;
        const double w1 = (2 * (f1 + nn) + 1) * pT;
        int idx = -1;
        if (first)
            idx = j + nn < N ? j + nn : -1;
        else if (j + nn - N < 0)
            idx = j + nn;
        else if (j + nn - N < N)
            idx = j + nn - N;
        const double2 v1 =
            hval(cw[0], dsum[0], d2sum[0], w1, idx >= 0, idx >= 0 ? X1[pidx(idx)] : make_double2(0, 0), 2 * (j + nn) + 1);
        const double w2 = (2 * f1 + 1) * pT;
        const double2 v2 = hval(cw[1], dsum[1], d2sum[1], w2, true, X2[pidx(j)], 2 * j + 1);
        acc[0] += cmul(cmul(green(f1), green(f1 + nn)), csub(v1, v2)).y;
    }
    block_sum<1>(acc, sums);
    if (tid == 0) {
        const double qn = 2.0 * nn * kPi * T;
        const int m = c % a.nbk;
        const double wt = (m == 0 || m == a.nbk - 1) ? 2.0 : 4.0;
        // Re[-i K acc] = K Im(acc)
        a.colv[(size_t)blockIdx.y * a.K4 + c] = a.U * T * a.nf * wt * a.dek[c] * sums[0] / (2.0 * qn);
    }
}

// out[row (1 + nbins) + 0] = sum_c colv[c], then per bin b the sum over the
// points of bin b; one block per value (x) and frequency (y), in a fixed order
// (strided compensated sums, shuffle tree, warps in order).
__global__ void __launch_bounds__(128) k_al_finish(const double *__restrict__ colv, const int *__restrict__ bin, int K4,
                                                   double *__restrict__ out) {
    __shared__ double tot[1];
    const int v = blockIdx.x;
    colv += (size_t)blockIdx.y * K4;
    KSum s;
    for (int c = threadIdx.x; c < K4; c += blockDim.x)
        if (v == 0 || (bin ? bin[c] : 0) == v - 1) s.add(colv[c]);
    KSum x[1] = {s};
    block_ksum<1>(x, tot);
    if (threadIdx.x == 0) out[(size_t)blockIdx.y * gridDim.x + v] = tot[0];
}

// ---------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------
template <int NBK>
struct RunAlHg {
    static cudaError_t run(const GridDev *g, const CondDev *c, const AlDev *a, const double *dG0p, double mu0,
                           double T, cudaStream_t st) {
        const size_t sm = SlicePlan<NBK>::bytes, smw = SliceSmem<NBK, SliceGroups<NBK>::wide>::bytes;
        cudaError_t e = set_smem(k_al_hg_slice<NBK>, sm);
        if (e != cudaSuccess) return e;
        if ((e = set_smem(k_al_hg_bound<NBK>, smw)) != cudaSuccess) return e;
        const double nf = 1.0 / ((double)g->nk0 * g->nk0);
        k_al_hg_slice<NBK><<<g->nw0 + 1, SlicePlan<NBK>::threads, sm, st>>>(c->tab, a->Grt, g->tw_k, g->nw0, g->n8, T, a->hGt,
                                                                   a->pre);
        if ((e = launched()) != cudaSuccess) return e;
        k_al_hg_bound<NBK><<<2, kSliceThreads, smw, st>>>(g->ek, c->dek, g->er, dG0p, a->Grt, g->tw_k, a->pre, g->nw0,
                                                          g->n8, mu0, T, nf, a->dhG);
        return launched();
    }
};

template <int N>
struct RunAlHgTau {
    static cudaError_t run(const GridDev *g, const AlDev *a, double T, cudaStream_t st) {
        const size_t sm = AlHgTauSmem<N>::bytes;
        cudaError_t e = set_smem(k_al_hg_tau<N>, sm);
        if (e != cudaSuccess) return e;
        k_al_hg_tau<N><<<a->K4p / 2, 256, sm, st>>>(a->hGt, a->dhG, g->spl_full, g->tw_w, g->ht_w, T, a->K4, a->hgq);
        return launched();
    }
};

template <int N>
struct RunAlHq {
    static cudaError_t run(const AlHqArgs *args, int npairs, int nf, cudaStream_t st) {
        const size_t sm = AlHqPlan<N>::smem;
        cudaError_t e = set_smem(k_al_hq<N>, sm);
        if (e != cudaSuccess) return e;
        k_al_hq<N><<<dim3(npairs, nf), AlHqPlan<N>::threads, sm, st>>>(*args);
        return launched();
    }
};

template <int NBK>
struct RunAlSlices {
    static cudaError_t run(const GridDev *g, const AlDev *a, const double *dG0p, double mu0, int nfr, cudaStream_t st) {
        const size_t sm = AlSlice<NBK>::bytes;
        cudaError_t e = set_smem(k_al_q2r<NBK>, sm);
        if (e != cudaSuccess) return e;
        if ((e = set_smem(k_al_r2k<NBK>, sm)) != cudaSuccess) return e;
        const double nf = 1.0 / ((double)g->nk0 * g->nk0);
        k_al_q2r<NBK><<<dim3(g->nw0 + 3, nfr), AlSlice<NBK>::threads, sm, st>>>(a->HQ, a->dHQ, g->tw_k, g->nw0, nf,
                                                                                  a->HR, a->dHR);
        if ((e = launched()) != cudaSuccess) return e;
        // (H(q, tau) is not read any more: G H(k, tau) takes its place)
        k_al_r2k<NBK><<<dim3(g->nw0 + 5, nfr), AlSlice<NBK>::threads, sm, st>>>(
            a->HR, a->dHR, a->Grt, g->er, dG0p, g->tw_k, g->nw0, g->n8, mu0, a->HQ, a->H2K, a->dHK);
        return launched();
    }
};

template <int N>
struct RunAlTau {
    static cudaError_t run(const AlTauArgs *args, int nf, cudaStream_t st) {
        const size_t sm = AlTauPlan<N>::smem;
        cudaError_t e = set_smem(k_al_tau<N>, sm);
        if (e != cudaSuccess) return e;
        k_al_tau<N><<<dim3(args->K4, nf), AlTauPlan<N>::threads, sm, st>>>(*args);
        return launched();
    }
};

}  // namespace

int al_batch(const GridDev &g, int K4, int nfreq) {
    // frequencies per launch: enough CTAs to fill the GPU several times over (the
    // k kernel has K4 a frequency), so that no half-empty last wave counts, as
    // long as the three arrays of a batch stay within a GB.  Whole call, 64^2 x
    // 1024 (96 frequencies): 10 a launch 14.2 ms, 5 15.1, 2 16.4, 1 18.9; 32^2 x
    // 256 (40): 14 a launch 1.2 ms, 2 2.0, 1 3.2.
    const size_t bytes = (size_t)3 * (g.nw0 + 1) * ((K4 + 1) & ~1) * sizeof(double2);
    const int fill = (sm_count() * 64 + K4 - 1) / K4, room = (int)std::max<size_t>(1, ((size_t)1 << 30) / bytes);
    return std::max(1, std::min({fill, room, nfreq, 40}));
}

cudaError_t launch_al_setup(const GridDev &g, const CondDev &c, const AlDev &a, const double *dG0p,
                            const double *chiq, const double *cinf, const double *cinf2, const double2 *S,
                            const double *s2, const double *s3, const double *sinf, double Usp, double Uch, double mu,
                            double mu0, double T, cudaStream_t st) {
    cudaError_t e = launch_gslice(g, a.Grt, mu0, T, st);
    if (e != cudaSuccess) return e;
    if ((e = dispatch_nbk<RunAlHg>(g.nbk, &g, &c, &a, dG0p, mu0, T, st)) != cudaSuccess) return e;
    if ((e = dispatch_nw<RunAlHgTau>(g.nw0, &g, &a, T, st)) != cudaSuccess) return e;
    AlTabArgs t;
    t.chiq = chiq;
    t.cinf = cinf;
    t.cinf2 = cinf2;
    t.hgq = a.hgq;
    t.S = S;
    t.s2 = s2;
    t.s3 = s3;
    t.sinf = sinf;
    t.ek = g.ek;
    t.tab = a.tab;
    t.shape = a.shape;
    t.dshape = a.dshape;
    t.gk = a.gk;
    t.K4 = a.K4;
    t.nbk = g.nbk;
    t.N = g.nw0;
    t.T = T;
    t.mu = mu;
    t.Usp = Usp;
    t.Uch = Uch;
    k_al_tables<<<a.K4, 128, 0, st>>>(t);
    return launched();
}

cudaError_t launch_al_freqs(const GridDev &g, const CondDev &c, const AlDev &a, const double *dG0p, int first, int count,
                            double U, double mu0, double T, cudaStream_t st) {
    if (count < 1 || count > a.batch) return cudaErrorInvalidValue;
    const int *ind = a.ind + first;
    AlHqArgs h;
    h.tab = a.tab;
    h.shape = a.shape;
    h.dshape = a.dshape;
    h.tw = g.tw_w;
    h.ht = g.ht_w;
    h.ind = ind;
    h.HQ = a.HQ;
    h.dHQ = a.dHQ;
    h.K4 = a.K4;
    h.K4p = a.K4p;
    h.T = T;
    cudaError_t e = dispatch_nw<RunAlHq>(g.nw0, &h, a.K4p / 2, count, st);
    if (e != cudaSuccess) return e;
    if ((e = dispatch_nbk<RunAlSlices>(g.nbk, &g, &a, dG0p, mu0, count, st)) != cudaSuccess) return e;
    AlTauArgs t;
    t.HK = a.HQ;
    t.H2K = a.H2K;
    t.dHK = a.dHK;
    t.gk = a.gk;
    t.dek = c.dek;
    t.spl = g.spl_full;
    t.tw = g.tw_w;
    t.ht = g.ht_w;
    t.ind = ind;
    t.colv = a.colv;
    t.K4 = a.K4;
    t.K4p = a.K4p;
    t.nbk = g.nbk;
    t.T = T;
    t.U = U;
    t.nf = 1.0 / ((double)g.nk0 * g.nk0);
    if ((e = dispatch_nw<RunAlTau>(g.nw0, &t, count, st)) != cudaSuccess) return e;
    k_al_finish<<<dim3(1 + a.nbins, count), 128, 0, st>>>(a.colv, a.nbins > 1 ? c.bin : nullptr, a.K4,
                                                          a.out + (size_t)first * (1 + a.nbins));
    return launched();
}

}  // namespace tpsc
