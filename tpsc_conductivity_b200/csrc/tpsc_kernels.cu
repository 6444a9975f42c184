// tpsc_kernels.cu -- sm_100a kernels of the TPSC hot path (FP64).
//
// Two kernel families do the transforms:
//  * slice kernels: one CTA per imaginary-time (or bosonic-frequency) slice.
//    The symmetric nbk x nbk quadrant of the slice lives in shared memory and
//    is transformed by a 2D DCT-I (tpsc_fft.cuh).  They replace the OpenMP
//    tau loops of chi0::calc_chiqw_FFT_spline (src/chi0.cpp:454-559),
//    chi::calc_chirt (src/chi.cpp:85-119) and green::calc_Self_FFT_spline
//    (src/green.cpp:1822-1892), which call FFTW REDFT00 per slice.
//  * tau kernels: one CTA per block of four octant columns.  The column data
//    (contiguous in the column-block layout) is staged in shared memory, the
//    clamped cubic spline along tau is solved in place, and the FFT of the
//    spline's third derivative gives the Matsubara values.  They replace the
//    per-q / per-k loops of src/chi0.cpp:586-690 and src/green.cpp:1925-2017
//    (LAPACK dgbsv + FFTW dft) and the 1D DCT-I over n of src/chi.cpp:129-144.
// Reductions (sum rules, traces) are two-pass and deterministic.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <set>
#include <utility>

#include "tpsc_device.cuh"
#include "tpsc_findzero.h"

namespace tpsc {

// kernels launched by this library (all contexts), for the instrumentation ABI
static std::atomic<long long> g_launches{0};

// tiling of the three tau transforms per N (process-wide; tpsc_tune_tau_tiles,
// tpsc_tune_tau_plans): 0 one column pair per CTA, radix-16 FFT passes;
// 1 four columns per CTA (k_*_tau); 2 one pair per CTA with radix-8 passes
// (k_*_tau2<N, 8>, N <= 2048; 0 elsewhere)
static std::atomic<int> g_tau_tile[4][13];
static std::atomic<long long> g_tau_tiles_version{0};
static int tile_index(int n) {
    int k = 0;
    while ((1 << k) < n && k < 12) ++k;
    return k;
}
int tau_tile(int kind, int n) { return g_tau_tile[kind][tile_index(n)].load(std::memory_order_relaxed); }
void set_tau_tile(int kind, int n, int tile) {
    if (g_tau_tile[kind][tile_index(n)].exchange(tile) != tile) g_tau_tiles_version.fetch_add(1);
}
long long tau_tiles_version() { return g_tau_tiles_version.load(); }
void bump_plans_version() { g_tau_tiles_version.fetch_add(1); }
// the same count for the calling host thread (kernels in one stream capture)
static thread_local long long t_launches = 0;
cudaError_t launched(int n) {
    g_launches.fetch_add(n, std::memory_order_relaxed);
    t_launches += n;
    return cudaGetLastError();
}

namespace {

// ---------------------------------------------------------------------------
// reductions: per-thread compensated (Kahan-Babuska) sums -> warp -> block ->
// per-block partials -> one block finishes in a fixed order
// ---------------------------------------------------------------------------

int grid_for(long long total, int threads) {
    long long b = (total + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > kMaxBlocks) b = kMaxBlocks;
    return (int)b;
}


// ---------------------------------------------------------------------------
// slice kernels
// ---------------------------------------------------------------------------

// Per-octant constants of G0(k, tau)/L^2 (src/green.cpp:1834-1837):
//   x = eps_k - mu0 > 0:  -exp(-tau x) / (exp(-x/T) + 1) / L^2
//   x <= 0:               -exp((beta - tau) x) / (exp(x/T) + 1) / L^2
// gk[o] = (x, prefactor), so one exp per element remains per slice.
__global__ void k_gk_table(const double *__restrict__ ek, int n8, double mu0, double T, double nk02,
                           double2 *__restrict__ gk, Bp b) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n8) return;
    ek = at(ek, b.arena);
    gk = at(gk, b.arena);
    mu0 = bpar(b, kPpMu0, mu0);
    T = bpar(b, kPpT, T);
    const double x = ek[o] - mu0;
    const double pre = x > 0 ? -1.0 / (exp(-x / T) + 1.0) / nk02 : -1.0 / (exp(x / T) + 1.0) / nk02;
    gk[o] = make_double2(x, pre);
}

// G(r, tau_j) = DCT-I[ G0(k, tau_j) / L^2 ], tau_j = j / (Nw0 T), j = 0..Nw0,
// with the overflow-safe branches of src/green.cpp:1834-1837.  The chi0 stage
// needs G(r, tau) and G(r, -tau) (src/chi0.cpp:462-495); G(r,-tau) =
// -G(r, beta - tau), so one table serves both stages.  Plain layout
// Grt[j * n8 + o].
template <int NBK, class P>
__global__ void __launch_bounds__(P::threads, P::blocks)
    k_gslice(const double2 *__restrict__ gk, const double2 *__restrict__ tw,
             int n8, int nw0, double T, double *__restrict__ Grt) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK, true>(S, tw);
    const int j = blockIdx.x;
    const double t = j / (nw0 * T);
    const double bt = 1.0 / T - t;
    fill_octant<NBK>(S, n8, [&](int o) -> double {
        const double2 c = __ldg(&gk[o]);
        return c.y * exp((c.x > 0 ? -t : bt) * c.x);
    });
    __syncthreads();
    plan_dct2<NBK, true>(S, tws);
    double *out = Grt + (size_t)j * n8;
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        out[o] = S[l * NBK + m];
    }
}

// chi0(r, tau_j) = -2 G(r, tau_j) G(r, -tau_j) and its DCT-I chi0(q, tau_j),
// j = 0..Nw0/2 (src/chi0.cpp:393-418, 497-517, 545-558).  tau = 0 uses
// G(r,0-) = G(r,0+) + delta_r0, tau = beta/2 uses 2 G^2.
template <int NBK, class P>
__global__ void __launch_bounds__(P::threads, P::blocks)
    k_chi0_slice(const double *__restrict__ Grt, const double2 *__restrict__ tw,
                 int n8, int nw0, double *__restrict__ chirt, double *__restrict__ chiq) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK, true>(S, tw);
    const int j = blockIdx.x;
    const int nb = nw0 / 2 + 1;
    // G(r, tau_j) and G(r, beta - tau_j) staged in the slice / scratch area
    static_assert(2 * StageRows<NBK>::drow_bytes <= P::tw_off, "inputs must fit");
    double *gp = S;
    double *gm = S + StageRows<NBK>::drow_bytes / sizeof(double);
    stage_drow<NBK>(gp, Grt + (size_t)j * n8);
    stage_drow<NBK>(gm, Grt + (size_t)(nw0 - j) * n8);
    cp_async_wait_all();
    __syncthreads();
    fill_from_staged<NBK, P::threads>(S, [&](int o) -> double {
        const double a = gp[o];
        double c;
        if (j == 0)
            c = (o == 0) ? -2.0 * a * (a + 1.0) : -2.0 * a * a;
        else if (j == nb - 1)
            c = 2.0 * a * a;
        else
            c = -2.0 * (-gm[o]) * a;
        chirt[bidx(j, o, nb)] = c;
        return c;
    });
    __syncthreads();
    plan_dct2<NBK, true>(S, tws);
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        chiq[bidx(j, o, nb)] = S[l * NBK + m];
    }
}

// d/dtau G(r,0+-) and d/dtau chi0(r,0), d/dtau chi0(q,0): the spline's left
// end condition (src/chi0.cpp:323-367, 420-447).  One CTA.
template <int NBK, class GT>
__global__ void __launch_bounds__(kSliceThreads, 1)
    k_chi0_boundary(const double *__restrict__ ek, const double *__restrict__ er,
                    const double2 *__restrict__ tw, const GT *__restrict__ Grt, int n8, double mu0, double T,
                    double nk02, double *__restrict__ dG0p, double *__restrict__ dtau_chirt0,
                    double *__restrict__ dtau_chiqt0, Bp b) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = slice_twiddles<NBK, SliceGroups<NBK>::wide>(S, tw);
    ek = at(ek, b.arena);
    er = at(er, b.arena);
    Grt = at(Grt, b.arena);
    dG0p = at(dG0p, b.arena);
    dtau_chirt0 = at(dtau_chirt0, b.arena);
    dtau_chiqt0 = at(dtau_chiqt0, b.arena);
    mu0 = bpar(b, kPpMu0, mu0);
    T = bpar(b, kPpT, T);
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        const double x = ek[o] - mu0;
        const double gkt = -1.0 / (exp(-x / T) + 1.0);
        put_sym<NBK>(S, l, m, -x * gkt / nk02);
    }
    __syncthreads();
    dct2_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    // every thread handles the same octant points in both loops, so the
    // first loop's S reads complete before its second-loop writes
    double dp_[(NBK * (NBK + 1) / 2 + kSliceThreads - 1) / kSliceThreads];
    double dc_[(NBK * (NBK + 1) / 2 + kSliceThreads - 1) / kSliceThreads];
    int k = 0;
    for (int o = threadIdx.x; o < n8; o += blockDim.x, ++k) {
        int l, m;
        oct_lm(o, l, m);
        const double dp = S[l * NBK + m];
        const double dm = ((o == 0) ? -mu0 : er[o]) - dp;
        const double g0 = Grt[o];
        const double dc = (o == 0) ? -2.0 * (dp * (1.0 + g0) + dm * g0) : -2.0 * (dp * g0 + dm * g0);
        dp_[k] = dp;
        dc_[k] = dc;
    }
    __syncthreads();
    k = 0;
    for (int o = threadIdx.x; o < n8; o += blockDim.x, ++k) {
        int l, m;
        oct_lm(o, l, m);
        dG0p[o] = dp_[k];
        dtau_chirt0[o] = dc_[k];
        put_sym<NBK>(S, l, m, dc_[k]);
    }
    __syncthreads();
    dct2_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        dtau_chiqt0[o] = S[l * NBK + m];
    }
}

// V(q, iqn) = (T/L^2) U [3 Usp (chisp - chi0) + Uch (chich - chi0)] / 8 and
// its DCT-I over q, one bosonic frequency per CTA (src/chi.cpp:89-115).
template <int NBK, class P>
__global__ void __launch_bounds__(P::threads, P::blocks)
    k_vertex_q(const double *__restrict__ chiq, const double2 *__restrict__ tw,
               int n8, int nb, double normFact, double U, const double *__restrict__ Usc, double *__restrict__ Vr) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK>(S, tw);
    const int j = blockIdx.x;
    const double Usp = Usc[0], Uch = Usc[1];
    // chi0(q, iq_j) staged in the slice / scratch area
    static_assert(StageRows<NBK>::blockrow_bytes <= P::tw_off, "inputs must fit");
    double *cs = S;
    stage_blockrow<NBK>(cs, chiq, j, nb);
    cp_async_wait_all();
    __syncthreads();
    fill_from_staged<NBK, P::threads>(S, [&](int o) -> double {
        const double c0 = cs[o];
        const double sp = c0 / (1.0 - Usp * c0 / 2.0);
        const double ch = c0 / (1.0 + Uch * c0 / 2.0);
        return normFact * U * (3.0 * Usp * (sp - c0) + Uch * (ch - c0)) / 8.0;
    });
    __syncthreads();
    plan_dct2<NBK>(S, tws);
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        Vr[bidx(j, o, nb)] = S[l * NBK + m];
    }
}

// d/dtau Sigma(k, 0) and d/dtau Sigma(k, beta): the spline end conditions of
// the self-energy (src/green.cpp:1743-1817).  Two CTAs, one 2D DCT-I each
// (blockIdx.x = 0: tau = 0, 1: tau = beta).
template <int NBK, class GT>
__global__ void __launch_bounds__(kSliceThreads, 1)
    k_sigma_boundary(const double *__restrict__ er, const double2 *__restrict__ tw,
                     const GT *__restrict__ Grt, const double *__restrict__ V, const double *__restrict__ dtau_chirt0,
                     const double *__restrict__ dG0p, int n8, int nw0, int n8p, double mu0, double U,
                     const double *__restrict__ Usc, double *__restrict__ dS, Bp b) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = slice_twiddles<NBK, SliceGroups<NBK>::wide>(S, tw);
    er = at(er, b.arena);
    Grt = at(Grt, b.arena);
    V = at(V, b.arena);
    dtau_chirt0 = at(dtau_chirt0, b.arena);
    dG0p = at(dG0p, b.arena);
    Usc = at(Usc, b.arena);
    dS = at(dS, b.arena);
    mu0 = bpar(b, kPpMu0, mu0);
    U = bpar(b, kPpU, U);
    const double fact = vertex_fact(U, Usc);
    const int nb = nw0 / 2 + 1;
    {
        const int side = blockIdx.x;
        const GT *g = Grt + (side == 0 ? 0 : (size_t)nw0 * n8);
        for (int o = threadIdx.x; o < n8; o += blockDim.x) {
            int l, m;
            oct_lm(o, l, m);
            const double v0 = V[bidx(0, o, nb)];
            double val;
            if (side == 0) {
                val = (fact * dtau_chirt0[o]) * g[o] + v0 * dG0p[o];
            } else {
                const double xi = (o == 0) ? -mu0 : er[o];
                val = (-fact * dtau_chirt0[o]) * g[o] + v0 * (-dG0p[o] + xi);
            }
            put_sym<NBK>(S, l, m, val);
        }
        __syncthreads();
        dct2_slice<NBK>(S, slice_scratch<NBK>(S), tws);
        for (int o = threadIdx.x; o < n8; o += blockDim.x) {
            int l, m;
            oct_lm(o, l, m);
            dS[side * n8p + o] = S[l * NBK + m];
        }
        __syncthreads();
    }
}

// Sigma(k, tau_j) = DCT-I[ G(r, tau_j) V(r, tau_j) ], j = 0..Nw0, with
// V(r, tau_j) = V(r, beta - tau_j) for tau_j > beta/2 (src/green.cpp:1822-1885),
// in FP64 (the mixed form's FP32 slice is k_sigma_slice32).
template <int NBK, class P>
__global__ void __launch_bounds__(P::threads, P::blocks)
    k_sigma_slice(const double *__restrict__ Grt, const double *__restrict__ V,
                  const double2 *__restrict__ tw, int n8, int nw0, int ahead, double *__restrict__ sigt) {
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK>(S, tw);
    const int j = blockIdx.x;
    const int nb = nw0 / 2 + 1;
    const int jv = j < nb ? j : nw0 - j;
    if (ahead > 0 && j + ahead <= nw0) {
        const int jn = j + ahead;
        prefetch_l2_range(Grt + (size_t)jn * n8, (size_t)n8 * sizeof(double));
        prefetch_l2_blockrow(V, jn < nb ? jn : nw0 - jn, nb, (n8 + 3) / 4);
    }
    // V(r, tau_j) and G(r, tau_j) staged in the slice / scratch area
    static_assert(StageRows<NBK>::blockrow_bytes + StageRows<NBK>::drow_bytes <= P::tw_off,
                  "inputs must fit");
    double *vs = S;
    double *gs = S + StageRows<NBK>::blockrow_bytes / sizeof(double);
    stage_blockrow<NBK>(vs, V, jv, nb);
    stage_drow<NBK>(gs, Grt + (size_t)j * n8);
    cp_async_wait_all();
    __syncthreads();
    fill_from_staged<NBK, P::threads>(S, [&](int o) -> double { return gs[o] * vs[o]; });
    __syncthreads();
    plan_dct2<NBK>(S, tws);
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        int l, m;
        oct_lm(o, l, m);
        sigt[bidx(j, o, nw0 + 1)] = S[l * NBK + m];
    }
}

// ---------------------------------------------------------------------------
// tau kernels
// ---------------------------------------------------------------------------

// chi0(q, iqn) from chi0(q, tau_j), j = 0..Nw0/2, for the four columns of one
// block, in place (src/chi0.cpp:586-690): clamped spline with slopes
// d/dtau chi0(q,0) and 0 at beta/2; FFT_{Nw0}[6 a_j antisymmetrised]
// (exp(+2 pi i jk/N)); chi0(q,0) = 2 * integral of the spline;
// chi0(q,iqn) = c2/qn^2 + [(1 - cos th) Re F + sin th Im F]/qn^4.
template <int N>
__global__ void __launch_bounds__(TauSmem<N>::threads, 1)
    k_chi0_tau(double *__restrict__ chiq, const double *__restrict__ dtau_chiqt0, double *__restrict__ chi0_inf,
               double *__restrict__ chi0_inf2, const double *__restrict__ spl, const double2 *__restrict__ tw,
               double T, int n8) {
    constexpr int NJ = N / 2 + 1;
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A + ((4 * NJ + 1) & ~1));
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + TauSmem<N>::tables_off(NJ));
    __shared__ double d0[4], dN[4], V0[4], VN[4], sV[4], sM[4], integ[4];
    const int o0 = 4 * blockIdx.x;
    double *g = chiq + (size_t)blockIdx.x * 4 * NJ;
    tau_tables(tw2, tw2 + 1, tw, tw, N);
    stage_in(A, g, NJ, n8 - o0);
    if (threadIdx.x < 4) {
        const int o = o0 + threadIdx.x;
        d0[threadIdx.x] = o < n8 ? dtau_chiqt0[o] : 0.0;
        dN[threadIdx.x] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        V0[threadIdx.x] = A[threadIdx.x * NJ];
        VN[threadIdx.x] = A[threadIdx.x * NJ + NJ - 1];
    }
    column_sums(A, NJ, 0, NJ, sV);
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_second_derivatives(A, NJ, NJ, h, d0, dN, spl, spl + NJ);
    column_sums(A, NJ, 0, NJ, sM);
    if (threadIdx.x < 4) {
        const int c = threadIdx.x;
        const double M0 = A[c * NJ], MN = A[c * NJ + NJ - 1];
        // sum_j [h (V_j + V_{j+1})/2 - h^3 (M_j + M_{j+1})/24]
        integ[c] = h * (sV[c] - 0.5 * (V0[c] + VN[c])) - h * h * h / 24.0 * (2.0 * sM[c] - M0 - MN);
    }
    __syncthreads();
    constexpr int G = FftPlan<N>::G;
#pragma unroll 1
    for (int pr = 0; pr < 2; ++pr) {
        const double *Ma = A + (2 * pr) * NJ;
        const double *Mb = A + (2 * pr + 1) * NJ;
        // FFT input: 6 a_j = (M_{j+1} - M_j)/h, antisymmetrised over [N/2, N)
        auto in = [&](int j) -> double2 {
            const bool lo = j < N / 2;
            const int jj = lo ? j : N - 1 - j;
            const double sg = lo ? 1.0 : -1.0;
            return make_double2(sg * (Ma[jj + 1] - Ma[jj]) * ih, sg * (Mb[jj + 1] - Mb[jj]) * ih);
        };
        if (threadIdx.x < G) group_fft_io<N, +1>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
        __syncthreads();
        for (int n = threadIdx.x + 1; n < NJ; n += blockDim.x) {
            const double2 Z = X[pidx(n)];
            const double2 Zc = X[pidx(N - n)];
            // split the packed transform: F_a = (Z_n + conj Z_{N-n})/2, F_b = (Z_n - conj Z_{N-n})/(2i)
            const double2 Fa = make_double2(0.5 * (Z.x + Zc.x), 0.5 * (Z.y - Zc.y));
            const double2 Fb = make_double2(0.5 * (Z.y + Zc.y), -0.5 * (Z.x - Zc.x));
            const double wn = 2 * n * kPi * T, iw = 1.0 / wn, i2 = iw * iw;
            const double2 w = tw_at(tw2, n);
            const double cth = w.x, sth = -w.y;  // cos, sin of 2 pi n / N
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = 2 * pr + q;
                const int o = o0 + c;
                const double2 F = q == 0 ? Fa : Fb;
                const double cinf = -2.0 * d0[c];
                double val = (cinf + ((1.0 - cth) * F.x + sth * F.y) * i2) * i2;
                if (o == 0) val = 0.0;
                A[c * NJ + n] = val;
                if (n == NJ - 1 && o < n8) chi0_inf2[o] = (o == 0) ? 0.0 : 2.0 * F.x;
            }
        }
        if (threadIdx.x < 2) A[(2 * pr + threadIdx.x) * NJ] = 2.0 * integ[2 * pr + threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x < 4) {
        const int o = o0 + threadIdx.x;
        if (o < n8) chi0_inf[o] = (o == 0) ? 0.0 : -2.0 * d0[threadIdx.x];
    }
    stage_out(A, g, NJ);
}

// V(r, tau_j) = DCT-I_n[ V(r, iqn) ] + U(3 Usp + Uch)/8 chi0(r, tau_j), in
// place on one column block (src/chi.cpp:129-166).
template <int N>
__global__ void __launch_bounds__(TauSmem<N>::threads, 1)
    k_vertex_tau(double *__restrict__ Vr, const double *__restrict__ chirt, const double2 *__restrict__ tw,
                 double U, const double *__restrict__ Usc, int n8) {
    constexpr int NJ = N / 2 + 1;
    const double fact = vertex_fact(U, Usc);
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A + ((4 * NJ + 1) & ~1));
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + TauSmem<N>::tables_off(NJ));
    double *g = Vr + (size_t)blockIdx.x * 4 * NJ;
    const double *cr = chirt + (size_t)blockIdx.x * 4 * NJ;
    tau_tables(tw2, tw2 + 1, tw, tw, N);
    stage_in(A, g, NJ, n8 - 4 * (int)blockIdx.x);
    __syncthreads();
    constexpr int G = FftPlan<N>::G;
#pragma unroll 1
    for (int pr = 0; pr < 2; ++pr) {
        double *a = A + (2 * pr) * NJ;
        double *b = A + (2 * pr + 1) * NJ;
        // even extension of the two columns: a DCT-I each, packed as Re/Im
        auto in = [&](int j) -> double2 {
            const int jj = j < NJ ? j : N - j;
            return make_double2(a[jj], b[jj]);
        };
        if (threadIdx.x < G) group_fft_io<N, -1>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
        __syncthreads();
        for (int n = threadIdx.x; n < NJ; n += blockDim.x) {
            const double2 Z = X[pidx(n)];
            a[n] = Z.x;
            b[n] = Z.y;
        }
        __syncthreads();
    }
    const int nvalid = n8 - 4 * (int)blockIdx.x;
    for (int i = threadIdx.x; i < 4 * NJ; i += blockDim.x)
        g[i] = (i & 3) < nvalid ? A[(i & 3) * NJ + (i >> 2)] + fact * cr[i] : 0.0;
}

// Sigma(k, i w_n) coefficients from Sigma(k, tau_j), j = 0..Nw0, for one
// column block (src/green.cpp:1935-2017): clamped spline with the two end
// slopes; F_n = sum_j exp(i pi j (2n+1)/N) 6 a_j (pre-twiddled FFT,
// exp(+2 pi i jk/N)); S_n = (1 - exp(i (2n+1) pi/N)) F_n for n < N/2.
// Sigma_inf2 = S'(0)+S'(beta), Sigma_inf3 = -(S''(0)+S''(beta)),
// Sigma_inf4 = Re S_{N/2-1}, Sigma_inf = -(S(0)+S(beta)) at k = 0.
template <int N>
__global__ void __launch_bounds__(TauSmem<N>::threads, 1)
    k_sigma_tau(const double *__restrict__ sigt, const double *__restrict__ dS, double2 *__restrict__ Sout,
                double *__restrict__ s2, double *__restrict__ s3, double *__restrict__ s4, double *__restrict__ sinf,
                const double *__restrict__ spl, const double2 *__restrict__ tw, const double2 *__restrict__ ht,
                double T, int n8, int n8p) {
    constexpr int NJ = N + 1;
    constexpr int NO = N / 2;
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A + ((4 * NJ + 1) & ~1));
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + TauSmem<N>::tables_off(NJ));
    const TwoLevelTw *ht2 = tw2 + 1;
    __shared__ double d0[4], dN[4];
    const int o0 = 4 * blockIdx.x;
    tau_tables(tw2, tw2 + 1, tw, ht, N);
    stage_in(A, sigt + (size_t)blockIdx.x * 4 * NJ, NJ, n8 - o0);
    if (threadIdx.x < 4) {
        const int o = o0 + threadIdx.x;
        d0[threadIdx.x] = dS[o];
        dN[threadIdx.x] = dS[n8p + o];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        const int o = o0 + threadIdx.x;
        if (o == 0) sinf[0] = -(A[0] + A[NJ - 1]);
        if (o < n8) s2[o] = d0[threadIdx.x] + dN[threadIdx.x];
    }
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_second_derivatives(A, NJ, NJ, h, d0, dN, spl, spl + NJ);
    if (threadIdx.x < 4) {
        const int o = o0 + threadIdx.x;
        const int c = threadIdx.x;
        if (o < n8) s3[o] = -(A[c * NJ] + A[c * NJ + N]);
    }
    constexpr int G = FftPlan<N>::G;
#pragma unroll 1
    for (int pr = 0; pr < 2; ++pr) {
        const double *Ma = A + (2 * pr) * NJ;
        const double *Mb = A + (2 * pr + 1) * NJ;
        // FFT input: exp(i pi j/N) 6 a_j, two columns packed as Re/Im
        auto in = [&](int j) -> double2 {
            const double fa = (Ma[j + 1] - Ma[j]) * ih;
            const double fb = (Mb[j + 1] - Mb[j]) * ih;
            return cmul(tw_at(ht2, j), make_double2(fa, fb));
        };
        if (threadIdx.x < G) group_fft_io<N, +1>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
        __syncthreads();
        for (int n = threadIdx.x; n < NO; n += blockDim.x) {
            const double2 Z = X[pidx(n)];
            const double2 Zr = X[pidx(N - 1 - n)];
            // F_a = (Z_n + conj Z_{N-1-n})/2, F_b = (Z_n - conj Z_{N-1-n})/(2i)
            const double2 Fa = make_double2(0.5 * (Z.x + Zr.x), 0.5 * (Z.y - Zr.y));
            const double2 Fb = make_double2(0.5 * (Z.y + Zr.y), -0.5 * (Z.x - Zr.x));
            const double2 e = tw_at(ht2, 2 * n + 1);
            const double2 f = make_double2(1.0 - e.x, -e.y);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = 2 * pr + q;
                const int o = o0 + c;
                const double2 Sv = cmul(f, q == 0 ? Fa : Fb);
                Sout[bidx(n, o, NO)] = Sv;
                if (n == NO - 1 && o < n8) s4[o] = Sv.x;
            }
        }
        __syncthreads();
    }
}

// Stage the two columns 2 half, 2 half + 1 of a four-column block (NJ rows)
// column-major into A; columns >= n8 as zeros.  Every element is an
// asynchronous 8-byte copy, all of a thread's copies in flight at once (the
// thread waits for its own; the caller's barrier publishes them).
__device__ __forceinline__ void stage_pair4(double *A, const double *blk4, int NJ, int half, int o0, int n8) {
    const bool c0 = o0 < n8, c1 = o0 + 1 < n8;
    const double *src = blk4 + 2 * half;
    for (int i = threadIdx.x; i < 2 * NJ; i += blockDim.x) {
        const int j = i >> 1, q = i & 1;
        double *dst = &A[q * NJ + j];
        if (q == 0 ? c0 : c1)
            cp_async8(dst, src + 4 * j + q);
        else
            *dst = 0.0;
    }
    cp_async_wait_all();
}

// The same transform for ONE pair of columns per CTA, two CTAs per SM: the
// pair is staged in a buffer of padded_len(N) complex and the FFT runs in
// place in it (its first pass reads the spline's third derivatives before the
// group barrier that precedes its writes), so a CTA needs ~74 KB of shared
// memory and at most 128 registers per thread.
template <int N>
struct Tau2Smem {
    static constexpr size_t buf = (size_t)padded_len(N) * sizeof(double2);
    static constexpr size_t bytes = buf + 2 * sizeof(TwoLevelTw);
};

template <int N, int EP = 16>
__global__ void __launch_bounds__(256, 2)
    k_sigma_tau2(const double *__restrict__ sigt, const double *__restrict__ dS, double2 *__restrict__ Sout,
                 double *__restrict__ s2, double *__restrict__ s3, double *__restrict__ s4, double *__restrict__ sinf,
                 const double *__restrict__ spl, const double2 *__restrict__ tw, const double2 *__restrict__ ht,
                 double T, int n8, int n8p, Bp b) {
    constexpr int NJ = N + 1;
    constexpr int NO = N / 2;
    static_assert(2 * NJ * sizeof(double) <= Tau2Smem<N>::buf, "pair must fit the FFT buffer");
    sigt = at(sigt, b.arena);
    dS = at(dS, b.arena);
    Sout = at(Sout, b.arena);
    s2 = at(s2, b.arena);
    s3 = at(s3, b.arena);
    s4 = at(s4, b.arena);
    sinf = at(sinf, b.arena);
    T = bpar(b, kPpT, T);
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A);
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + Tau2Smem<N>::buf);
    const TwoLevelTw *ht2 = tw2 + 1;
    __shared__ double d0[2], dN[2];
    const int pair = blockIdx.x, blk = pair >> 1, half = pair & 1;
    const int o0 = 2 * pair;
    // the end slopes, read before the staging wait
    double d0r = 0.0, dNr = 0.0;
    if (threadIdx.x < 2) {
        d0r = dS[o0 + threadIdx.x];
        dNr = dS[n8p + o0 + threadIdx.x];
    }
    tau_tables(tw2, tw2 + 1, tw, ht, N);
    // the pair's two columns of the four-column block, column-major
    stage_pair4(A, sigt + (size_t)blk * 4 * NJ, NJ, half, o0, n8);
    if (threadIdx.x < 2) {
        d0[threadIdx.x] = d0r;
        dN[threadIdx.x] = dNr;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        const int o = o0 + threadIdx.x;
        if (o == 0) sinf[0] = -(A[0] + A[NJ - 1]);
        if (o < n8) s2[o] = d0[threadIdx.x] + dN[threadIdx.x];
    }
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_second_derivatives<2>(A, NJ, NJ, h, d0, dN, spl, spl + NJ);
    if (threadIdx.x < 2) {
        const int o = o0 + threadIdx.x;
        if (o < n8) s3[o] = -(A[threadIdx.x * NJ] + A[threadIdx.x * NJ + N]);
    }
    constexpr int G = FftPlan<N, EP>::G;
    static_assert(G <= 256, "one FFT group of at most 256 threads");
    if (threadIdx.x < G) {
        const double *Ma = A, *Mb = A + NJ;
        auto in = [&](int j) -> double2 {
            const double fa = (Ma[j + 1] - Ma[j]) * ih;
            const double fb = (Mb[j + 1] - Mb[j]) * ih;
            return cmul(tw_at(ht2, j), make_double2(fa, fb));
        };
        group_fft_io<N, +1, false, true, EP>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
    }
    __syncthreads();
    for (int n = threadIdx.x; n < NO; n += blockDim.x) {
        const double2 Z = X[pidx(n)];
        const double2 Zr = X[pidx(N - 1 - n)];
        const double2 Fa = make_double2(0.5 * (Z.x + Zr.x), 0.5 * (Z.y - Zr.y));
        const double2 Fb = make_double2(0.5 * (Z.y + Zr.y), -0.5 * (Z.x - Zr.x));
        const double2 e = tw_at(ht2, 2 * n + 1);
        const double2 f = make_double2(1.0 - e.x, -e.y);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int o = o0 + q;
            const double2 Sv = cmul(f, q == 0 ? Fa : Fb);
            Sout[bidx(n, o, NO)] = Sv;
            if (n == NO - 1 && o < n8) s4[o] = Sv.x;
        }
    }
}

// k_chi0_tau for one pair per CTA (in-place FFT, two CTAs per SM); results
// go straight back to chiq.
template <int N, int EP = 16>
__global__ void __launch_bounds__(256, 2)
    k_chi0_tau2(double *__restrict__ chiq, const double *__restrict__ dtau_chiqt0, double *__restrict__ chi0_inf,
                double *__restrict__ chi0_inf2, const double *__restrict__ spl, const double2 *__restrict__ tw,
                double T, int n8, Bp b) {
    constexpr int NJ = N / 2 + 1;
    chiq = at(chiq, b.arena);
    dtau_chiqt0 = at(dtau_chiqt0, b.arena);
    chi0_inf = at(chi0_inf, b.arena);
    chi0_inf2 = at(chi0_inf2, b.arena);
    T = bpar(b, kPpT, T);
    static_assert(2 * NJ * sizeof(double) <= Tau2Smem<N>::buf, "pair must fit the FFT buffer");
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A);
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + Tau2Smem<N>::buf);
    __shared__ double d0[2], dN[2], V0[2], VN[2], sV[2], sM[2], integ[2];
    const int pair = blockIdx.x, blk = pair >> 1, half = pair & 1;
    const int o0 = 2 * pair;
    double *g = chiq + (size_t)blk * 4 * NJ + 2 * half;
    // the left end slope, read before the staging wait
    const double d0r = (threadIdx.x < 2 && o0 + (int)threadIdx.x < n8) ? dtau_chiqt0[o0 + threadIdx.x] : 0.0;
    tau_tables(tw2, tw2 + 1, tw, tw, N);
    stage_pair4(A, chiq + (size_t)blk * 4 * NJ, NJ, half, o0, n8);
    if (threadIdx.x < 2) {
        d0[threadIdx.x] = d0r;
        dN[threadIdx.x] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        V0[threadIdx.x] = A[threadIdx.x * NJ];
        VN[threadIdx.x] = A[threadIdx.x * NJ + NJ - 1];
    }
    column_sums<2>(A, NJ, 0, NJ, sV);
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_second_derivatives<2>(A, NJ, NJ, h, d0, dN, spl, spl + NJ);
    column_sums<2>(A, NJ, 0, NJ, sM);
    if (threadIdx.x < 2) {
        const int c = threadIdx.x;
        const double M0 = A[c * NJ], MN = A[c * NJ + NJ - 1];
        integ[c] = h * (sV[c] - 0.5 * (V0[c] + VN[c])) - h * h * h / 24.0 * (2.0 * sM[c] - M0 - MN);
    }
    constexpr int G = FftPlan<N, EP>::G;
    static_assert(G <= 256, "one FFT group of at most 256 threads");
    if (threadIdx.x < G) {
        const double *Ma = A, *Mb = A + NJ;
        auto in = [&](int j) -> double2 {
            const bool lo = j < N / 2;
            const int jj = lo ? j : N - 1 - j;
            const double sg = lo ? 1.0 : -1.0;
            return make_double2(sg * (Ma[jj + 1] - Ma[jj]) * ih, sg * (Mb[jj + 1] - Mb[jj]) * ih);
        };
        group_fft_io<N, +1, false, true, EP>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
    }
    __syncthreads();
    for (int n = threadIdx.x + 1; n < NJ; n += blockDim.x) {
        const double2 Z = X[pidx(n)];
        const double2 Zc = X[pidx(N - n)];
        const double2 Fa = make_double2(0.5 * (Z.x + Zc.x), 0.5 * (Z.y - Zc.y));
        const double2 Fb = make_double2(0.5 * (Z.y + Zc.y), -0.5 * (Z.x - Zc.x));
        const double wn = 2 * n * kPi * T, iw = 1.0 / wn, i2 = iw * iw;
        const double2 w = tw_at(tw2, n);
        const double cth = w.x, sth = -w.y;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int o = o0 + q;
            const double2 F = q == 0 ? Fa : Fb;
            const double cinf = -2.0 * d0[q];
            double val = (cinf + ((1.0 - cth) * F.x + sth * F.y) * i2) * i2;
            if (o == 0) val = 0.0;
            g[4 * n + q] = val;
            if (n == NJ - 1 && o < n8) chi0_inf2[o] = (o == 0) ? 0.0 : 2.0 * F.x;
        }
    }
    if (threadIdx.x < 2) {
        const int o = o0 + threadIdx.x;
        g[threadIdx.x] = 2.0 * integ[threadIdx.x];
        if (o < n8) chi0_inf[o] = (o == 0) ? 0.0 : -2.0 * d0[threadIdx.x];
    }
}

// k_vertex_tau for one pair per CTA (in-place FFT, two CTAs per SM).
template <int N, int EP = 16>
__global__ void __launch_bounds__(256, 2)
    k_vertex_tau2(double *__restrict__ Vr, const double *__restrict__ chirt, const double2 *__restrict__ tw,
                  double U, const double *__restrict__ Usc, int n8, Bp b) {
    constexpr int NJ = N / 2 + 1;
    Vr = at(Vr, b.arena);
    chirt = at(chirt, b.arena);
    Usc = at(Usc, b.arena);
    U = bpar(b, kPpU, U);
    const double fact = vertex_fact(U, Usc);
    static_assert(2 * NJ * sizeof(double) <= Tau2Smem<N>::buf, "pair must fit the FFT buffer");
    extern __shared__ __align__(16) double A[];
    double2 *X = reinterpret_cast<double2 *>(A);
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(A) + Tau2Smem<N>::buf);
    const int pair = blockIdx.x, blk = pair >> 1, half = pair & 1;
    const int o0 = 2 * pair;
    tau_tables(tw2, tw2 + 1, tw, tw, N);
    stage_pair4(A, Vr + (size_t)blk * 4 * NJ, NJ, half, o0, n8);
    __syncthreads();
    constexpr int G = FftPlan<N, EP>::G;
    static_assert(G <= 256, "one FFT group of at most 256 threads");
    if (threadIdx.x < G) {
        const double *a = A, *b = A + NJ;
        // even extension of the two columns: a DCT-I each, packed as Re/Im
        auto in = [&](int j) -> double2 {
            const int jj = j < NJ ? j : N - j;
            return make_double2(a[jj], b[jj]);
        };
        group_fft_io<N, -1, false, true, EP>(X, threadIdx.x, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X});
    }
    __syncthreads();
    double *g = Vr + (size_t)blk * 4 * NJ + 2 * half;
    // the pair's chi0(r, tau) values of a row are 16 contiguous bytes
    const double2 *cr = reinterpret_cast<const double2 *>(chirt + (size_t)blk * 4 * NJ + 2 * half);
    for (int n = threadIdx.x; n < NJ; n += blockDim.x) {
        const double2 Z = X[pidx(n)];
        const double2 c = __ldcs(&cr[2 * n]);
        g[4 * n] = (o0 < n8) ? Z.x + fact * c.x : 0.0;
        g[4 * n + 1] = (o0 + 1 < n8) ? Z.y + fact * c.y : 0.0;
    }
}

// ---------------------------------------------------------------------------
// tau transforms by groups: a pair of columns is one complex column in a buffer
// of its own, splined (spline_complex) and transformed in place by one FFT group
// of G = N/16 threads; a CTA of 128 threads takes 128/G pairs, so that every
// thread transforms whatever N is, and its barriers are the groups' own.  Pair
// kernels of 256 threads (k_*_tau2) leave all but N/16 of them idle in the
// transform and sweep columns of 65 nodes in chunks of one row with 30 warm-up
// rows.  64 points of the parameter sweep, one launch: chi0 at
// Nw0 = 256 189 -> 39 us, Sigma 183 -> 39, at 1024 256 -> 115 and 253 -> 132;
// 128^2 x 2048: chi0 58 -> 45, Sigma 65 -> 55, V 30 -> 26.  At Nw0 = 4096, where
// the pair kernels' 256 threads all transform, they stay: Sigma 380 us against
// 399, chi0 306 against 316, V 182 against 189 (half the threads sweep here).
// They also stay for a launch whose pairs they hold at once (tau_groups): there
// only the time of one pair counts, and the more threads have the shorter chains.
// One point, group -> pair kernel: 16^2 x 64 V 10.0 -> 5.3 us, Sigma 16.7 -> 12.1,
// chi0 15.5 -> 12.7; 64^2 x 1024 V 11.7 -> 8.2, Sigma 20.3 -> 15.8, chi0 18.2 -> 15.0.
// ---------------------------------------------------------------------------
constexpr int kTau3Max = 2048;
template <int N>
struct Tau3Plan {
    static constexpr int G = FftPlan<N>::G;
    static constexpr int threads = 128;
    static constexpr int pairs = threads / G;  // of a CTA
    static constexpr int blocks = 4;           // of an SM
    static_assert(G <= threads, "one pair needs at most the block");
    static constexpr int x_len = padded_len(N) + 2;        // N + 1 nodes
    static constexpr size_t tables_off = (size_t)pairs * x_len * sizeof(double2);
    static constexpr size_t bytes = tables_off + 2 * sizeof(TwoLevelTw);
};
template <int N>
struct Tau3Group {
    double2 *X;
    TwoLevelTw *tw2;  // FFT twiddles, then the half-step ones
    int grp, t, pair;
    __device__ explicit Tau3Group(double2 *smem) {
        using P = Tau3Plan<N>;
        grp = threadIdx.x / P::G;
        t = threadIdx.x % P::G;
        pair = blockIdx.x * P::pairs + grp;
        X = smem + grp * P::x_len;
        tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(smem) + P::tables_off);
    }
    // the pair's two columns (NJ rows) of their four-column block; columns from n8 on as zeros
    __device__ void load(const double *a, int NJ, int n8) {
        const double *src = a + (size_t)(pair >> 1) * 4 * NJ + 2 * (pair & 1);
        for (int j = t; j < NJ; j += Tau3Plan<N>::G) cp_async16(&X[pidx(j)], src + 4 * (size_t)j);
        cp_async_wait_all();
        if (2 * pair + 1 >= n8)
            for (int j = t; j < NJ; j += Tau3Plan<N>::G) {
                const double2 v = X[pidx(j)];
                X[pidx(j)] = make_double2(2 * pair < n8 ? v.x : 0.0, 0.0);
            }
    }
    __device__ void sync() { group_sync<Tau3Plan<N>::G>(grp); }
    // sums of a and c over the group's threads, in its thread 0; red: one entry per warp of the block
    __device__ double2 sum(KSum a, KSum c, double4 *red) {
        constexpr int G = Tau3Plan<N>::G, W = G < 32 ? G : 32;
        const unsigned lanes = G < 32 ? ((1u << W) - 1u) << ((threadIdx.x & 31) / W * W) : 0xffffffffu;
        a.join_lanes<W>(lanes);
        c.join_lanes<W>(lanes);
        if constexpr (G > 32) {
            if (t % 32 == 0) red[threadIdx.x / 32] = make_double4(a.s, a.c, c.s, c.c);
            sync();
            if (t == 0)
                for (int w = 1; w < G / 32; ++w) {
                    const double4 r = red[threadIdx.x / 32 + w];
                    a.join(r.x, r.y);
                    c.join(r.z, r.w);
                }
            sync();
        }
        return make_double2(a.value(), c.value());
    }
};
// the two columns of a packed transform at bins n and its partner
__device__ __forceinline__ void store_pair(double *g, double a, double b) {
    *reinterpret_cast<double2 *>(g) = make_double2(a, b);
}

// k_sigma_tau by groups
template <int N>
__global__ void __launch_bounds__(Tau3Plan<N>::threads, Tau3Plan<N>::blocks)
    k_sigma_tau3(const double *__restrict__ sigt, const double *__restrict__ dS, double2 *__restrict__ Sout,
                 double *__restrict__ s2, double *__restrict__ s3, double *__restrict__ s4, double *__restrict__ sinf,
                 const double *__restrict__ spl, const double2 *__restrict__ tw, const double2 *__restrict__ ht,
                 double T, int n8, int n8p, Bp b) {
    constexpr int NJ = N + 1, NO = N / 2, G = Tau3Plan<N>::G;
    sigt = at(sigt, b.arena);
    dS = at(dS, b.arena);
    Sout = at(Sout, b.arena);
    s2 = at(s2, b.arena);
    s3 = at(s3, b.arena);
    s4 = at(s4, b.arena);
    sinf = at(sinf, b.arena);
    T = bpar(b, kPpT, T);
    extern __shared__ __align__(16) double2 smem3[];
    Tau3Group<N> q(smem3);
    tau_tables(q.tw2, q.tw2 + 1, tw, ht, N);
    __syncthreads();
    const int o0 = 2 * q.pair;
    if (o0 >= n8p) return;
    const TwoLevelTw *ht2 = q.tw2 + 1;
    double2 *X = q.X;
    const double2 d0 = make_double2(dS[o0], dS[o0 + 1]), dN = make_double2(dS[n8p + o0], dS[n8p + o0 + 1]);
    q.load(sigt, NJ, n8);
    q.sync();
    if (q.t == 0) {
        const double2 v0 = X[0], vN = X[pidx(N)];
        if (o0 == 0) sinf[0] = -(v0.x + vN.x);
        if (o0 < n8) s2[o0] = d0.x + dN.x;
        if (o0 + 1 < n8) s2[o0 + 1] = d0.y + dN.y;
    }
    q.sync();
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    spline_complex<N>(X, NJ, q.t, q.grp, h, d0, dN, spl, spl + NJ);
    if (q.t == 0) {
        const double2 m0 = X[0], mN = X[pidx(N)];
        if (o0 < n8) s3[o0] = -(m0.x + mN.x);
        if (o0 + 1 < n8) s3[o0 + 1] = -(m0.y + mN.y);
    }
    auto in = [&](int j) -> double2 {
        const double2 u = X[pidx(j)], v = X[pidx(j + 1)];
        return cmul(tw_at(ht2, j), make_double2((v.x - u.x) * ih, (v.y - u.y) * ih));
    };
    group_fft_io<N, +1, false, true>(X, q.t, (const TwoLevelTw *)q.tw2, q.grp, in, ScratchIO{X});
    q.sync();
    for (int n = q.t; n < NO; n += G) {
        double2 Fa, Fb;
        split_real(X[pidx(n)], X[pidx(N - 1 - n)], Fa, Fb);
        const double2 e = tw_at(ht2, 2 * n + 1);
        const double2 f = make_double2(1.0 - e.x, -e.y);
        const double2 Sa = cmul(f, Fa), Sb = cmul(f, Fb);
        Sout[bidx(n, o0, NO)] = Sa;
        Sout[bidx(n, o0 + 1, NO)] = Sb;
        if (n == NO - 1) {
            if (o0 < n8) s4[o0] = Sa.x;
            if (o0 + 1 < n8) s4[o0 + 1] = Sb.x;
        }
    }
}

// k_chi0_tau by groups (the mixed form's: its sums are taken in another order
// than k_chi0_tau2's, see launch_chi0_tau)
template <int N>
__global__ void __launch_bounds__(Tau3Plan<N>::threads, Tau3Plan<N>::blocks)
    k_chi0_tau3(double *__restrict__ chiq, const double *__restrict__ dtau_chiqt0, double *__restrict__ chi0_inf,
                double *__restrict__ chi0_inf2, const double *__restrict__ spl, const double2 *__restrict__ tw,
                double T, int n8, int n8p, Bp b) {
    constexpr int NO = N / 2, NJ = NO + 1, G = Tau3Plan<N>::G;
    chiq = at(chiq, b.arena);
    dtau_chiqt0 = at(dtau_chiqt0, b.arena);
    chi0_inf = at(chi0_inf, b.arena);
    chi0_inf2 = at(chi0_inf2, b.arena);
    T = bpar(b, kPpT, T);
    extern __shared__ __align__(16) double2 smem3[];
    __shared__ double4 red[Tau3Plan<N>::threads / 32];
    Tau3Group<N> q(smem3);
    tau_tables(q.tw2, q.tw2 + 1, tw, tw, N);
    __syncthreads();
    const int o0 = 2 * q.pair;
    if (o0 >= n8p) return;
    double2 *X = q.X;
    const double2 d0 =
        make_double2(o0 < n8 ? dtau_chiqt0[o0] : 0.0, o0 + 1 < n8 ? dtau_chiqt0[o0 + 1] : 0.0);
    const double2 zero = make_double2(0.0, 0.0);
    q.load(chiq, NJ, n8);
    q.sync();
    // trapezoid sums of the nodes and of the second derivatives
    auto trapezoid = [&]() -> double2 {
        KSum a, c;
        for (int j = q.t; j < NJ; j += G) {
            const double2 v = X[pidx(j)];
            const double w = (j == 0 || j == NO) ? 0.5 : 1.0;
            a.add(w * v.x);
            c.add(w * v.y);
        }
        return q.sum(a, c, red);
    };
    const double h = 1.0 / (N * T), ih = 1.0 / h;
    const double2 sV = trapezoid();
    q.sync();
    spline_complex<N>(X, NJ, q.t, q.grp, h, d0, zero, spl, spl + NJ);
    const double2 sM = trapezoid();
    q.sync();
    auto in = [&](int j) -> double2 {
        const bool lo = j < NO;
        const int jj = lo ? j : N - 1 - j;
        const double sg = lo ? ih : -ih;
        const double2 u = X[pidx(jj)], v = X[pidx(jj + 1)];
        return make_double2((v.x - u.x) * sg, (v.y - u.y) * sg);
    };
    group_fft_io<N, +1, false, true>(X, q.t, (const TwoLevelTw *)q.tw2, q.grp, in, ScratchIO{X});
    q.sync();
    double *g = chiq + (size_t)(q.pair >> 1) * 4 * NJ + 2 * (q.pair & 1);
    for (int n = q.t + 1; n < NJ; n += G) {
        double2 Fa, Fb;
        split_real(X[pidx(n)], X[pidx(N - n)], Fa, Fb);
        const double wn = 2 * n * kPi * T, iw = 1.0 / wn, i2 = iw * iw;
        const double2 w = tw_at(q.tw2, n);
        const double cth = w.x, sth = -w.y;
        const double va = (-2.0 * d0.x + ((1.0 - cth) * Fa.x + sth * Fa.y) * i2) * i2;
        const double vb = (-2.0 * d0.y + ((1.0 - cth) * Fb.x + sth * Fb.y) * i2) * i2;
        store_pair(g + 4 * n, o0 == 0 ? 0.0 : va, vb);
        if (n == NJ - 1) {
            if (o0 < n8) chi0_inf2[o0] = o0 == 0 ? 0.0 : 2.0 * Fa.x;
            if (o0 + 1 < n8) chi0_inf2[o0 + 1] = 2.0 * Fb.x;
        }
    }
    if (q.t == 0) {
        const double h3 = h * h * h / 12.0;
        store_pair(g, 2.0 * (h * sV.x - h3 * sM.x), 2.0 * (h * sV.y - h3 * sM.y));
        if (o0 < n8) chi0_inf[o0] = o0 == 0 ? 0.0 : -2.0 * d0.x;
        if (o0 + 1 < n8) chi0_inf[o0 + 1] = -2.0 * d0.y;
    }
}

// k_vertex_tau by groups
template <int N>
__global__ void __launch_bounds__(Tau3Plan<N>::threads, Tau3Plan<N>::blocks)
    k_vertex_tau3(double *__restrict__ Vr, const double *__restrict__ chirt, const double2 *__restrict__ tw, double U,
                  const double *__restrict__ Usc, int n8, int n8p, Bp b) {
    constexpr int NJ = N / 2 + 1, G = Tau3Plan<N>::G;
    Vr = at(Vr, b.arena);
    chirt = at(chirt, b.arena);
    Usc = at(Usc, b.arena);
    U = bpar(b, kPpU, U);
    const double fact = vertex_fact(U, Usc);
    extern __shared__ __align__(16) double2 smem3[];
    Tau3Group<N> q(smem3);
    tau_tables(q.tw2, q.tw2 + 1, tw, tw, N);
    __syncthreads();
    const int o0 = 2 * q.pair;
    if (o0 >= n8p) return;
    double2 *X = q.X;
    q.load(Vr, NJ, n8);
    q.sync();
    // even extension of the two columns: a DCT-I each, packed as Re/Im
    auto in = [&](int j) -> double2 { return X[pidx(j < NJ ? j : N - j)]; };
    group_fft_io<N, -1, false, true>(X, q.t, (const TwoLevelTw *)q.tw2, q.grp, in, ScratchIO{X});
    q.sync();
    const size_t off = (size_t)(q.pair >> 1) * 4 * NJ + 2 * (q.pair & 1);
    double *g = Vr + off;
    const double2 *cr = reinterpret_cast<const double2 *>(chirt + off);
    for (int n = q.t; n < NJ; n += G) {
        const double2 Z = X[pidx(n)];
        const double2 c = __ldcs(&cr[2 * n]);
        store_pair(g + 4 * n, o0 < n8 ? Z.x + fact * c.x : 0.0, o0 + 1 < n8 ? Z.y + fact * c.y : 0.0);
    }
}

// ---------------------------------------------------------------------------
// sum rules and traces
// ---------------------------------------------------------------------------

// Deterministic grid reduction for the column-block reducers: every block
// stores NV partial sums, the last block to arrive (ticket counter) adds all
// partials in block order with compensated summation and resets the ticket.
// Partials are read with ld.global.cg, so the other blocks' stores (fenced
// before the ticket increment) are seen.
template <int NV>
__device__ void grid_finish(double (&v)[NV], Reduce r, double offset0) {
    __shared__ double red[32][NV];
    __shared__ bool last;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double x = 0.0;
            for (int w = 0; w < nw; ++w) x += red[w][k];
            r.partial[k * kMaxBlocks + blockIdx.x] = x;
        }
        __threadfence();
        const unsigned t = atomicAdd(r.ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // warp k adds value k over the blocks: lane-strided compensated sums and a
    // shuffle tree, a fixed order (deterministic)
    const int nb = gridDim.x;
    for (int k = warp; k < NV; k += blockDim.x >> 5) {
        KSum acc;
        for (int b = lane; b < nb; b += 32) acc.add(__ldcg(&r.partial[k * kMaxBlocks + b]));
        double x = acc.value();
        for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if (lane == 0) r.result[k] = x + (k == 0 ? offset0 : 0.0);
    }
    if (threadIdx.x == 0) *r.ticket = 0u;
}

constexpr int kRedThreads = 256;

// chi::traceDiffChispChi0 (sgn = -1) / traceDiffChichChi0 (sgn = +1)
// (src/chi.cpp:738-830): sum over q and n <= Nw0/2 of w T/Nq [chi/(1 + sgn U
// chi/2) - chi], plus the tail Nw0/2 < n <= Nw0 with chi = c2/qn^2 + c4/qn^4,
// and d/dU of the same sum.  One CTA per block of four octant columns: the
// block's rows are contiguous 32-byte loads.  w16 holds the octant weights
// (16 halved on edges and diagonal; 0 on padding columns); the row n = 0
// carries an extra factor 1/2.
// Stored frequencies j < jdir are summed term by term (jdir = nb: all of
// them); the Newton form passes jdir < nb and adds the frequencies above as a
// power series in h from the moments of k_chi0_moments.
__global__ void __launch_bounds__(kRedThreads)
    k_sumrule(const double4 *__restrict__ chiq, const double *__restrict__ cinf, const double *__restrict__ cinf2,
              const double *__restrict__ w16, const double *__restrict__ tailq, int nb, int jdir, int tail, double Uv,
              double sgn, double T, double scale, Reduce r) {
    const int blk = blockIdx.x;
    const double hu = sgn * Uv / 2.0;
    const double4 w = *reinterpret_cast<const double4 *>(w16 + 4 * blk);
    const double ww[4] = {w.x, w.y, w.z, w.w};
    double v, dv, tv = 0.0, tdv = 0.0;
    sumrule_stored<true>(chiq, ww, blk, nb, jdir, hu, v, dv);
    if (tail)
        sumrule_tail(cinf, cinf2, ww, blk, nb, hu, sgn, T, tv, tdv, [&](int, double a, double b, double &f, double &df) {
            tail_series(a, b, hu, tailq, f, df);
        });
    dv *= -0.5 * sgn;
    double out[2] = {scale * (v + tv), scale * (dv + tdv)};
    grid_finish<2>(out, r, 0.0);
}

// Directional derivative of k_sumrule's trace at fixed U (jdir = nb, tail
// term by term) in the direction (dchi, dchi0_inf, dchi0_inf2):
//   sum w T/Nq [1/(1 + h chi)^2 - 1] dchi,  h = sgn U/2,
// with the same weights (n = 0 halved) and the same tail frequencies, for both sum
// rules (h = -Usp/2 -> result[0], Uch/2 -> result[1]): chi and dchi, and the tail's
// divisions, once for the two.  Bound: the dependent divisions of a few rows a
// thread; 128^2 x 2048: 2 x 16.4 us -> 19.4 us.
__global__ void __launch_bounds__(kRedThreads)
    k_sumrule_tan(const double4 *__restrict__ chiq, const double4 *__restrict__ dchiq,
                  const double *__restrict__ cinf, const double *__restrict__ cinf2, const double *__restrict__ dcinf,
                  const double *__restrict__ dcinf2, const double *__restrict__ w16, int nb, double Usp, double Uch,
                  double T, double scale, Reduce r) {
    const double hu[2] = {-Usp / 2.0, Uch / 2.0};
    double v[2] = {0.0, 0.0};
    const int blk = blockIdx.x;
    const int o0 = 4 * blk;
    const double4 w = *reinterpret_cast<const double4 *>(w16 + o0);
    const double ww[4] = {w.x, w.y, w.z, w.w};
    const double4 *col = chiq + (size_t)blk * nb, *dcol = dchiq + (size_t)blk * nb;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        const double4 x = col[j], dx = dcol[j];
        const double f = j == 0 ? 0.5 : 1.0;
        const double xs[4] = {x.x, x.y, x.z, x.w}, ds[4] = {dx.x, dx.y, dx.z, dx.w};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            double s = 0.0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double q = 1.0 / (1.0 + hu[i] * xs[c]);
                s += ww[c] * (q * q - 1.0) * ds[c];
            }
            v[i] += f * s;
        }
    }
    const int nwmax = nb - 1;
    const double tw = 2.0 * 3.141592653589793 * T;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (ww[c] == 0.0) continue;
        const double a = cinf[o0 + c], b = cinf2[o0 + c], da = dcinf[o0 + c], db = dcinf2[o0 + c];
        for (int t = threadIdx.x; t < nwmax; t += blockDim.x) {
            const double wn = (nwmax + 1 + t) * tw;
            const double i2 = 1.0 / (wn * wn);
            const double xv = a * i2 + b * i2 * i2, dxv = da * i2 + db * i2 * i2;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double q = 1.0 / (1.0 + hu[i] * xv);
                v[i] += ww[c] * (q * q - 1.0) * dxv;
            }
        }
    }
    double out[2] = {scale * v[0], scale * v[1]};
    grid_finish<2>(out, r, 0.0);
}

// The Newton form's sum-rule evaluation: only the stored frequencies
// j < jdir (the rest enters as the moment series on the host), over a
// flattened (column block, j) index so that every thread has independent
// loads in flight; a short grid.
__global__ void __launch_bounds__(kRedThreads)
    k_sumrule_low(const double4 *__restrict__ chiq, const double *__restrict__ w16, int nb, int nblk, int jdir,
                  double Uv, double sgn, double scale, Reduce r) {
    const double hu = sgn * Uv / 2.0;
    double v = 0.0, dv = 0.0;
    const long long total = (long long)nblk * jdir;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < total;
         it += (long long)gridDim.x * blockDim.x) {
        const int blk = (int)(it / jdir), j = (int)(it - (long long)blk * jdir);
        const double4 x = ld_stream4(&chiq[(size_t)blk * nb + j]);
        const double4 w = reinterpret_cast<const double4 *>(w16)[blk];
        const double f = j == 0 ? 0.5 : 1.0;
        const double xs[4] = {x.x, x.y, x.z, x.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double q = xs[c] / (1.0 + hu * xs[c]);
            v += f * ww[c] * (q - xs[c]);
            dv += f * ww[c] * q * q;
        }
    }
    double out[2] = {scale * v, scale * (-0.5 * sgn) * dv};
    grid_finish<2>(out, r, 0.0);
}


// Per-frequency moments of chi0 for the sum-rule series of the Newton form:
// mom[j][k] = sum_q w_q f_j chi(q, iq_j)^(k+2), k < kMomP (f_0 = 1/2, else 1),
// and cmax[j] = max_q |chi(q, iq_j)|.  One block per frequency j, a fixed
// reduction order (deterministic).  With |h chi| < kMomSeriesMax for every
// q at frequencies j >= jdir,
//   sum_{q, j >= jdir} w f [chi/(1 + h chi) - chi] = sum_{m=1}^{kMomP} (-h)^m M_{m+1}
// up to a relative (kMomSeriesMax)^kMomP.
__global__ void __launch_bounds__(256)
    k_chi0_moments(const double4 *__restrict__ chiq, const double *__restrict__ w16, int nb, int nblk,
                   double *__restrict__ mom, double *__restrict__ cmax, Bp b) {
    const int j = blockIdx.x;
    chiq = at(chiq, b.arena);
    mom = at(mom, b.arena);
    cmax = at(cmax, b.arena);
    const double f = j == 0 ? 0.5 : 1.0;
    double acc[kMomP + 1];
#pragma unroll
    for (int k = 0; k <= kMomP; ++k) acc[k] = 0.0;
    double mx = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        const double4 x = chiq[(size_t)b * nb + j];
        const double4 w = *reinterpret_cast<const double4 *>(w16 + 4 * b);
        const double xs[4] = {x.x, x.y, x.z, x.w}, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (ws[c] == 0.0) continue;
            const double v = xs[c];
            mx = fmax(mx, fabs(v));
            double pw = ws[c] * f * v * v;
#pragma unroll
            for (int k = 0; k < kMomP; ++k) {
                acc[k] += pw;
                pw *= v;
            }
        }
    }
    acc[kMomP] = mx;
    __shared__ double red[8][kMomP + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k <= kMomP; ++k)
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_down_sync(0xffffffffu, acc[k], off);
            acc[k] = (k == kMomP) ? fmax(acc[k], o) : acc[k] + o;
        }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k <= kMomP; ++k) red[warp][k] = acc[k];
    __syncthreads();
    if (threadIdx.x <= kMomP) {
        const int k = threadIdx.x;
        double x = red[0][k];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) x = (k == kMomP) ? fmax(x, red[w][k]) : x + red[w][k];
        if (k == kMomP)
            cmax[j] = x;
        else
            mom[(size_t)j * kMomP + k] = x;
    }
}

// Moments of the Matsubara tail of the sum rule (n = Nw0/2+1 .. Nw0, where
// chi0 = a/qn^2 + b/qn^4, a = chi0_inf, b = chi0_inf2): per column the
// U-independent S_p = sum_n chi_n^p from the power sums Q_k = sum_n qn^-2k,
// S_p = sum_i C(p,i) a^(p-i) b^i Q_(p+i), weighted and summed over the
// columns -> partial for block_store, value k = sum w S_(k+2), k < kMomP, and
// value kMomP = max over columns of |chi| at the first tail frequency.
__global__ void __launch_bounds__(256)
    k_tail_moments(const double *__restrict__ cinf, const double *__restrict__ cinf2, const double *__restrict__ w16,
                   const double *__restrict__ tailq, int n8, int nb, double T, double *partial, Bp b) {
    constexpr int NV = kMomP + 1;
    cinf = at(cinf, b.arena);
    cinf2 = at(cinf2, b.arena);
    tailq = at(tailq, b.arena);
    partial = at(partial, b.arena);
    T = bpar(b, kPpT, T);
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    const int nwmax = nb - 1;
    const double wn1 = (nwmax + 1) * 2.0 * 3.141592653589793 * T;
    const double x1 = 1.0 / (wn1 * wn1);
    for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < n8; o += gridDim.x * blockDim.x) {
        const double w = w16[o];
        if (w == 0.0) continue;
        const double a = cinf[o], b = cinf2[o];
        double ap[2 * kMomP + 2], bp[2 * kMomP + 2];
        ap[0] = bp[0] = 1.0;
#pragma unroll
        for (int k = 1; k < kMomP + 2; ++k) {
            ap[k] = ap[k - 1] * a;
            bp[k] = bp[k - 1] * b;
        }
#pragma unroll
        for (int m = 1; m <= kMomP; ++m) {
            const int p = m + 1;
            double Sp = 0.0, coef = 1.0;
#pragma unroll
            for (int i = 0; i <= p; ++i) {
                Sp += coef * ap[p - i] * bp[i] * __ldg(&tailq[p + i]);
                coef = coef * (p - i) / (i + 1);
            }
            acc[m - 1] += w * Sp;
        }
        acc[kMomP] = fmax(acc[kMomP], fabs(a) * x1 + fabs(b) * x1 * x1);
    }
    // the max enters block_store's sum: keep it in a separate shared slot
    __shared__ double mx[32];
    double m = acc[kMomP];
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) mx[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double x = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) x = fmax(x, mx[i]);
        partial[(2 * kMomP + 1) * kMaxBlocks + blockIdx.x] = x;
    }
    acc[kMomP] = 0.0;
    block_store<NV>(acc, partial);
}

// Tr(G - G0) at chemical potential pmu (green::traceDiffG,
// src/green.cpp:3108-3182): stored frequencies j < Nw0/2 with the full Sigma,
// tail Nw0/2 <= j <= Nw0 with its asymptotic form.  One CTA per column block.

// Stored frequencies j < jdir term by term (jdir = Nw0/2: all), and the
// tail Nw0/2 <= j <= Nw0 when `tail` is set; the Newton form covers the
// rest with the series of k_sigma_moments.
// DERIV = false: the value alone.
template <bool DERIV>
__global__ void __launch_bounds__(kRedThreads)
    k_trace_diff_G(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                   const double *__restrict__ s4, const double *__restrict__ sinfp, const double *__restrict__ ek,
                   const double *__restrict__ w16, int nw0, double mu0, double pmu, double T, int jdir, int tail,
                   Reduce r) {
    double out[1 + DERIV], v, dv;
    trace_diff_block<true>(S, s2, s3, s4, sinfp, ek, w16, blockIdx.x, nw0, mu0, pmu, T, jdir, tail, v, dv);
    out[0] = v;
    if (DERIV) out[DERIV] = dv;
    grid_finish<1 + DERIV>(out, r, 0.0);
}

// The Newton form's Tr(G - G0) evaluation: only the stored frequencies
// j < jdir, over a flattened (column block, j) index, a short grid.
__global__ void __launch_bounds__(kRedThreads)
    k_trace_diff_G_low(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                       const double *__restrict__ sinfp, const double *__restrict__ ek,
                       const double *__restrict__ w16, int nw0, int nblk, double mu0, double pmu, double T, int jdir,
                       Reduce r) {
    const int NO = nw0 / 2;
    const double sinf = sinfp[0];
    const double pt = 3.141592653589793 * T;
    double v = 0.0, dv = 0.0;
    const long long total = (long long)nblk * jdir;
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < total;
         it += (long long)gridDim.x * blockDim.x) {
        const int blk = (int)(it / jdir), j = (int)(it - (long long)blk * jdir);
        const int o0 = 4 * blk;
        const double4 *row = reinterpret_cast<const double4 *>(S + (size_t)blk * 4 * NO);
        const double4 p = ld_stream4(&row[2 * j]), q = ld_stream4(&row[2 * j + 1]);
        const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                               make_double2(q.z, q.w)};
        const double wn = (2 * j + 1) * pt, i1 = 1.0 / wn;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double w = __ldg(&w16[o0 + c]);
            if (w == 0.0) continue;
            double rS, iS;
            sigma_full(i1, sinf, __ldg(&s2[o0 + c]), __ldg(&s3[o0 + c]), sv[c], rS, iS);
            trdiff_term(wn, rS, iS, __ldg(&ek[o0 + c]), mu0, pmu, w, v, dv);
        }
    }
    double out[2] = {v, dv};
    grid_finish<2>(out, r, 0.0);
}

// Tr Sigma G0 and its asymptotic correction (green::traceSelfG,
// src/green.cpp:3001-3084); w8 = w16 / 2.
__global__ void __launch_bounds__(kRedThreads)
    k_trace_self_G(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                   const double *__restrict__ sinfp, const double *__restrict__ ek, const double *__restrict__ w16,
                   int nw0, double mu0, double T, double nk02, Reduce r) {
    const int blk = blockIdx.x, o0 = 4 * blk, NO = nw0 / 2;
    const double sinf = sinfp[0];
    const double pt = 3.141592653589793 * T;
    KSum v, v2;
    const double4 *row = reinterpret_cast<const double4 *>(S + (size_t)blk * 4 * NO);
    for (int j = threadIdx.x; j < NO; j += blockDim.x) {
        const double wn = (2 * j + 1) * pt;
        const double i1 = 1.0 / wn;
        const double4 p = ld_stream4(&row[2 * j]), q = ld_stream4(&row[2 * j + 1]);
        const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                               make_double2(q.z, q.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double w8 = 0.5 * w16[o0 + c];
            if (w8 == 0.0) continue;
            double rS, iS;
            sigma_full(i1, sinf, s2[o0 + c], s3[o0 + c], sv[c], rS, iS);
            const double x = ek[o0 + c] - mu0;
            const double tmp = w8 * T * 2 / (nk02 * (wn * wn + x * x));
            v.add(tmp * (rS * (-x) + iS * wn));
            v2.add(w8 * sinf * T * 2 / (nk02 * (wn * wn + x * x)));
        }
    }
    if (threadIdx.x < 4) {
        const int c = threadIdx.x;
        const double w8 = 0.5 * w16[o0 + c];
        if (w8 != 0.0) {
            const double x = ek[o0 + c] - mu0;
            if (fabs(x) > 1.0e-12) {
                v2.add(w8 * sinf * (1.0 / (exp(x / T) + 1.0) - 0.5) / x / nk02);
            } else {
                const double ex = (x < 0) ? exp(x / T) : exp(-x / T);
                v2.add(-w8 * sinf * ex / ((ex + 1.0) * (ex + 1.0) * nk02 * T));
            }
        }
    }
    double out[2] = {v.value(), v2.value()};
    grid_finish<2>(out, r, 0.0);
}

// Tr Sigma G (green::traceSelfG2, src/green.cpp:2929-2976) by itself, for the searches
// that the host drives
__global__ void __launch_bounds__(kRedThreads)
    k_trace_self_G2(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                    const double *__restrict__ sinfp, const double *__restrict__ ek, const double *__restrict__ w16,
                    int nw0, double mu, double T, double nk02, Reduce r) {
    double out[1] = {trace_self2_block<true>(S, s2, s3, sinfp, ek, w16, blockIdx.x, nw0, mu, T, nk02)};
    grid_finish<1>(out, r, 0.0);
}

// raw and tail parts of chi0::traceChi0 (src/chi0.cpp:1498-1584)
__global__ void __launch_bounds__(kRedThreads)
    k_trace_chi0(const double4 *__restrict__ chiq, const double *__restrict__ cinf, const double *__restrict__ cinf2,
                 const double *__restrict__ w16, int nb, double T, double Nq, Reduce r) {
    const int blk = blockIdx.x, o0 = 4 * blk, nwmax = nb - 1;
    const double4 w = *reinterpret_cast<const double4 *>(w16 + o0);
    const double ww[4] = {w.x, w.y, w.z, w.w};
    KSum v, vt;
    const double4 *col = chiq + (size_t)blk * nb;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        const double4 x = col[j];
        const double f = (j == 0 || j == nwmax) ? 0.5 : 1.0;
        const double xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (ww[c] != 0.0) v.add(f * ww[c] * T * xs[c] / Nq);
    }
    for (int t = threadIdx.x; t < nwmax - 1; t += blockDim.x) {
        const double wn = 2 * 3.141592653589793 * (nwmax + 1 + t) * T;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (ww[c] != 0.0)
                vt.add(ww[c] * T * (cinf[o0 + c] / (wn * wn) + cinf2[o0 + c] / (wn * wn * wn * wn)) / Nq);
    }
    double out[2] = {v.value(), vt.value()};
    grid_finish<2>(out, r, 0.0);
}

// chi0max and its wave vector (src/chi0.cpp:703-717): the reference scans l
// and then m downwards keeping the first strict maximum, i.e. among equal
// maxima the largest l, then the largest m.  That is the maximum of the
// total order (value, l, m), so any reduction tree gives the reference's
// point: per-thread scans, then shuffle trees.  One block.
struct MaxPt {
    double v;
    int l, m;
};
__device__ __forceinline__ bool better(const MaxPt &a, const MaxPt &b) {
    return a.v > b.v || (a.v == b.v && (a.l > b.l || (a.l == b.l && a.m > b.m)));
}
__device__ __forceinline__ MaxPt max_shfl(MaxPt a, int off) {
    MaxPt b;
    b.v = __shfl_down_sync(0xffffffffu, a.v, off);
    b.l = __shfl_down_sync(0xffffffffu, a.l, off);
    b.m = __shfl_down_sync(0xffffffffu, a.m, off);
    return better(b, a) ? b : a;
}
__global__ void __launch_bounds__(1024)
    k_chi0max(const double *__restrict__ chiq, int n8, int nb, double *result, Bp b) {
    chiq = at(chiq, b.arena);
    result = at(result, b.arena);
    // values <= 0 never win: the reference's scan starts from chi0max = 0.
    // Each round issues its U loads before any comparison (one latency per
    // round instead of one per point).
    constexpr int U = 4;
    MaxPt best{0.0, -1, -1};
    for (int o0 = threadIdx.x; o0 < n8; o0 += U * blockDim.x) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * (int)blockDim.x;
            v[u] = o < n8 ? chiq[bidx(0, o, nb)] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * (int)blockDim.x;
            if (o >= n8) continue;
            int l, m;
            oct_lm(o, l, m);
            const MaxPt c{v[u], l, m};
            if (c.v > 0.0 && better(c, best)) best = c;
        }
    }
    for (int off = 16; off > 0; off >>= 1) best = max_shfl(best, off);
    __shared__ MaxPt w[32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x < 32) {
        best = threadIdx.x < (int)(blockDim.x >> 5) ? w[threadIdx.x] : MaxPt{0.0, -1, -1};
        for (int off = 16; off > 0; off >>= 1) best = max_shfl(best, off);
        if (threadIdx.x == 0) {
            result[0] = best.l < 0 ? 0.0 : best.v;
            result[1] = best.l < 0 ? 0 : best.l;
            result[2] = best.m < 0 ? 0 : best.m;
        }
    }
}

// mu0 of the finite lattice by safeguarded Newton on the density
// n(mu) = sum_o w 2 f(eps_o - mu) / L^2 (the function of green0::find_mu /
// ddensity_mu_PBC, src/green0.cpp:182-262) in one block: each iteration is a
// block reduction of n(mu) - n and dn/dmu in a fixed order; the Newton step
// is kept inside the bracket [-8, 8] that the sign of n - n0 shrinks, a
// bisection otherwise; stops when the step is below 1e-15 (1 + |mu|).
// The Newton form's replacement of the reference's root search.
__global__ void __launch_bounds__(1024)
    k_mu0_newton(const double *__restrict__ ek, int n8, int nbk, double n, double T,
                 double nk2, double *result, Bp b) {
    __shared__ double red[32][2];
    __shared__ double s_mu;
    __shared__ int s_done, s_it;
    ek = at(ek, b.arena);
    result = at(result, b.arena);
    n = bpar(b, kPpN, n);
    T = bpar(b, kPpT, T);
    // a batched launch writes the point's mu0 into its scalars (half filling
    // without t', t'': 0, no search)
    double *mu0_out = b.pp ? at(const_cast<double *>(b.pp), b.arena) + kPpMu0 : nullptr;
    if (mu0_out && at(b.pp, b.arena)[kPpMu0Fixed] != 0.0) {
        if (threadIdx.x == 0) {
            *mu0_out = 0.0;
            result[0] = 0.0;
            result[1] = 0.0;
        }
        return;
    }
    double lo = -8.0, hi = 8.0, mu = 0.0;
    if (threadIdx.x == 0) {
        s_mu = 0.0;
        s_done = 0;
    }
    __syncthreads();
    for (int it = 0; it < 200; ++it) {
        mu = s_mu;
        double v = 0.0, dv = 0.0;
        for (int o = threadIdx.x; o < n8; o += blockDim.x) {
            int l, m;
            oct_lm(o, l, m);
            const int w = oct_weight(8, l, m, nbk);
            const double f = 1.0 / (exp((ek[o] - mu) / T) + 1.0);
            v += 2 * w * f / nk2;
            dv += 2 * w * f * (1.0 - f) / (T * nk2);
        }
        for (int off = 16; off > 0; off >>= 1) {
            v += __shfl_down_sync(0xffffffffu, v, off);
            dv += __shfl_down_sync(0xffffffffu, dv, off);
        }
        if ((threadIdx.x & 31) == 0) {
            red[threadIdx.x >> 5][0] = v;
            red[threadIdx.x >> 5][1] = dv;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double V = 0.0, D = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                V += red[w][0];
                D += red[w][1];
            }
            const double F = V - n;
            if (F > 0)
                hi = mu;
            else
                lo = mu;
            double mn = (D > 0) ? mu - F / D : 0.5 * (lo + hi);
            if (!(mn > lo && mn < hi)) mn = 0.5 * (lo + hi);
            const bool done = F == 0.0 || fabs(mn - mu) <= 1e-15 * (1.0 + fabs(mu));
            s_mu = done && F == 0.0 ? mu : mn;
            s_done = done;
            s_it = it + 1;
        }
        __syncthreads();
        if (s_done) break;
    }
    if (threadIdx.x == 0) {
        result[0] = s_mu;
        result[1] = s_it;
        if (mu0_out) *mu0_out = s_mu;
    }
}

// ---------------------------------------------------------------------------
// real-frequency continuation on Matsubara samples of Sigma
// ---------------------------------------------------------------------------
constexpr int kPadeMax = 32;

// Per octant k: Sigma(k, z_j) at z_j = i (2 n_j + 1) pi T with the stored
// frequency j (green::MDC and find_FS_inter read Self_kw_array at j while
// z_j uses n[j], src/green.cpp:992, 2276), then either
//  mode 0: Vidberg-Serene continued-fraction Pade (pade_cont_frac_coef_rec
//          and pade, src/generique.cpp:1605-1663) at the Nz energies z;
//  mode 1: Lagrange polynomial through the Nn samples (src/green.cpp:2297-2299).
// out_sig [N8][Nz] (complex, may be null), out_A [N8][Nz] with
// A = -Im 1/(z - (eps_k - mu) - Sigma)/pi.
// One CTA per octant point: the samples and (mode 0) the continued-fraction
// coefficients in shared memory -- the recursion runs over l in parallel, one
// barrier per order m -- then the CTA's threads take the energies z.  Each
// (k, z) value is the same arithmetic as a one-thread evaluation.
__global__ void __launch_bounds__(128)
    k_pade_sigma(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                 const double *__restrict__ sinfp, const double *__restrict__ ek, const int *__restrict__ nidx,
                 int Nn, const double2 *__restrict__ z, int Nz, int mode, int n8, int nw0, double mu, double T,
                 double2 *__restrict__ out_sig, double *__restrict__ out_A) {
    const int o = blockIdx.x;
    const int NO = nw0 / 2;
    __shared__ double2 f[kPadeMax], x0[kPadeMax], g[kPadeMax], coef[kPadeMax];
    const int t = threadIdx.x;
    if (t < Nn) {
        const double sinf = sinfp[0];
        x0[t] = make_double2(0.0, (2 * nidx[t] + 1) * 3.141592653589793 * T);
        const double wn = (2 * t + 1) * 3.141592653589793 * T;
        const double i1 = 1.0 / wn, i2 = i1 * i1, i4 = i2 * i2;
        const double2 Sv = S[bidx(t, o, NO)];
        // Sigma(k, i w_j) = Sinf/z + C2/z^2 + C3/z^3 + S/z^4 at z = i w_j
        f[t] = make_double2(-s2[o] * i2 + Sv.x * i4, -sinf * i1 + s3[o] * i2 * i1 + Sv.y * i4);
        g[t] = f[t];
    }
    __syncthreads();
    if (mode == 0) {
        // continued-fraction coefficients: g_0(l) = f_l,
        // g_m(l) = (g_{m-1}(m-1) - g_{m-1}(l)) / ((x_l - x_{m-1}) g_{m-1}(l)), coef_m = g_m(m)
        if (t == 0) coef[0] = g[0];
        for (int m = 1; m < Nn; ++m) {
            const double2 gm = g[m - 1];
            if (t >= m && t < Nn) {
                const double2 dx = make_double2(x0[t].x - x0[m - 1].x, x0[t].y - x0[m - 1].y);
                g[t] = cdiv(csub(gm, g[t]), cmul(dx, g[t]));
            }
            __syncthreads();
            if (t == 0) coef[m] = g[m];
        }
        __syncthreads();
    }
    const double e = ek[o] - mu;
    for (int iz = t; iz < Nz; iz += blockDim.x) {
        const double2 zz = z[iz];
        double2 sig;
        if (mode == 0) {
            double2 A = make_double2(1.0, 0.0);
            double2 B = cadd(make_double2(1.0, 0.0), cmul(csub(zz, x0[0]), coef[1]));
            double2 q = cdiv(A, B);
            for (int j = 3; j <= Nn; ++j) {
                const double2 tj = cmul(csub(zz, x0[j - 2]), coef[j - 1]);
                A = cadd(make_double2(1.0, 0.0), cdiv(tj, A));
                B = cadd(make_double2(1.0, 0.0), cdiv(tj, B));
                q = cdiv(cmul(q, A), B);
            }
            sig = cmul(q, coef[0]);
        } else {
            sig = make_double2(0.0, 0.0);
            for (int j = 0; j < Nn; ++j) {
                double2 term = f[j];
                for (int i = 0; i < Nn; ++i)
                    if (i != j) term = cmul(term, cdiv(csub(zz, x0[i]), csub(x0[j], x0[i])));
                sig = cadd(sig, term);
            }
        }
        const double2 d = make_double2(zz.x - e - sig.x, zz.y - sig.y);
        const double2 gz = cdiv(make_double2(1.0, 0.0), d);
        if (out_sig) out_sig[(size_t)o * Nz + iz] = sig;
        out_A[(size_t)o * Nz + iz] = -gz.y / 3.141592653589793;
    }
}

// green::Gwn_local (src/green.cpp:209-266): G_loc(i w_j) = sum_k w/L^2
// 1/(z - eps_k + mu - Sigma(k, z)), w = 8 halved on edges and diagonal.
// One block per frequency j.
__global__ void k_gwn_local(const double2 *__restrict__ S, const double *__restrict__ s2,
                            const double *__restrict__ s3, const double *__restrict__ sinfp,
                            const double *__restrict__ ek, const double *__restrict__ w16, int n8, int nw0, double mu,
                            double T, double nk02, double2 *__restrict__ out) {
    const int j = blockIdx.x, NO = nw0 / 2;
    const double sinf = sinfp[0];
    const double wn = (2 * j + 1) * 3.141592653589793 * T;
    const double i1 = 1.0 / wn, i2 = i1 * i1, i4 = i2 * i2;
    double re = 0.0, im = 0.0;
    for (int o = threadIdx.x; o < n8; o += blockDim.x) {
        const double2 Sv = S[bidx(j, o, NO)];
        const double rS = -s2[o] * i2 + Sv.x * i4;
        const double iS = -sinf * i1 + s3[o] * i2 * i1 + Sv.y * i4;
        const double2 g = cdiv(make_double2(0.5 * w16[o] / nk02, 0.0),
                               make_double2(-ek[o] + mu - rS, wn - iS));
        re += g.x;
        im += g.y;
    }
    __shared__ double sr[1024], si[1024];
    sr[threadIdx.x] = re;
    si[threadIdx.x] = im;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = 0; i < (int)blockDim.x; ++i) {
            a += sr[i];
            b += si[i];
        }
        out[j] = make_double2(a, b);
    }
}

// blocked -> [j][o]
__global__ void k_unblock(const double *__restrict__ src, double *__restrict__ dst, int NJ, int nrows, int n8) {
    const long long total = (long long)nrows * n8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i / n8), o = (int)(i % n8);
        dst[i] = src[bidx(j, o, NJ)];
    }
}
__global__ void k_unblock_c(const double2 *__restrict__ src, double2 *__restrict__ dst, int NJ, int nrows, int n8) {
    const long long total = (long long)nrows * n8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i / n8), o = (int)(i % n8);
        dst[i] = src[bidx(j, o, NJ)];
    }
}

// The full Sigma(k, i w_n) = Sinf/z + C2/z^2 + C3/z^3 + S/z^4, z = i w_n,
// w_n = (2n+1) pi T, n < NO, formed in FP64 and rounded to FP32, [n][o]
// (the mixed form's copy-out: S alone could not be rounded, its 1/z^4 term
// cancels against the others at low n)
__global__ void k_sigma_full32(const double2 *__restrict__ S, const double *__restrict__ s2,
                               const double *__restrict__ s3, const double *__restrict__ sinfp, int NO, int n8,
                               double T, float2 *__restrict__ dst) {
    const long long total = (long long)NO * n8;
    const double sinf = sinfp[0];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int n = (int)(i / n8), o = (int)(i % n8);
        double rS, iS;
        sigma_full(1.0 / ((2 * n + 1) * kPi * T), sinf, s2[o], s3[o], S[bidx(n, o, NO)], rS, iS);
        dst[i] = make_float2((float)rS, (float)iS);
    }
}

// [j][o] -> blocked (NJ rows): the setters' inverse of k_unblock
__global__ void k_block(const double *__restrict__ src, double *__restrict__ dst, int NJ, int nrows, int n8) {
    const long long total = (long long)nrows * n8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i / n8), o = (int)(i % n8);
        dst[bidx(j, o, NJ)] = src[i];
    }
}
__global__ void k_block_c(const double2 *__restrict__ src, double2 *__restrict__ dst, int NJ, int nrows, int n8) {
    const long long total = (long long)nrows * n8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i / n8), o = (int)(i % n8);
        dst[bidx(j, o, NJ)] = src[i];
    }
}

// row j of a blocked (NJ rows) array -> dst[o]
__global__ void k_take_row(const double *__restrict__ src, int NJ, int j, int n8, double *__restrict__ dst) {
    for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < n8; o += gridDim.x * blockDim.x)
        dst[o] = src[bidx(j, o, NJ)];
}

__global__ void k_gather(GatherPieces p, unsigned *__restrict__ dst) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int k = 0; k < p.n; ++k)
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < p.words[k]; i += stride)
            dst[p.dst[k] + i] = p.src[k][i];
}

struct StoreVals {
    double v[4];
    int n;
};
__global__ void k_store(StoreVals s, double *__restrict__ dst) {
    if ((int)threadIdx.x < s.n) dst[threadIdx.x] = s.v[threadIdx.x];
}

// ---------------------------------------------------------------------------
// launch wrappers per compiled size
// ---------------------------------------------------------------------------
template <int NBK>
struct RunGslice {
    static cudaError_t run(const GridDev *g, double *Grt, double mu0, double T, cudaStream_t st) {
        const double nk02 = (double)g->nk0 * g->nk0;
        k_gk_table<<<(g->n8 + 255) / 256, 256, 0, st>>>(g->ek, g->n8, mu0, T, nk02, g->gk, Bp{});
        cudaError_t e = launched();
        if (e != cudaSuccess) return e;
        return with_plan<NBK, SlicePlan<NBK, true>, 1>(g->nw0 + 1, [&](auto plan) {
            using P = decltype(plan);
            cudaError_t err = set_smem(k_gslice<NBK, P>, P::bytes);
            if (err != cudaSuccess) return err;
            k_gslice<NBK, P><<<g->nw0 + 1, P::threads, P::bytes, st>>>(g->gk, g->tw_k, g->n8, g->nw0, T, Grt);
            return launched();
        });
    }
};
template <int NBK>
struct RunChi0Boundary {
    template <class GT>
    static cudaError_t run(const GridDev *g, const GT *Grt, double mu0, double T, double *dG0p, double *dchirt0,
                           double *dchiqt0, const Bp *b, cudaStream_t st) {
        const size_t smw = SliceSmem<NBK, SliceGroups<NBK>::wide>::bytes;
        cudaError_t e = set_smem(k_chi0_boundary<NBK, GT>, smw);
        if (e != cudaSuccess) return e;
        const double nk02 = (double)g->nk0 * g->nk0;
        k_chi0_boundary<NBK, GT><<<dim3(1, 1, b->P), kSliceThreads, smw, st>>>(g->ek, g->er, g->tw_k, Grt, g->n8, mu0,
                                                                               T, nk02, dG0p, dchirt0, dchiqt0, *b);
        return launched();
    }
};
template <int NBK>
struct RunChi0Slice {
    static cudaError_t run(const GridDev *g, const double *Grt, double *chirt, double *chiq, cudaStream_t st) {
        return with_plan<NBK, SlicePlan<NBK, true>, 1>(g->nb, [&](auto plan) {
            using P = decltype(plan);
            cudaError_t e = set_smem(k_chi0_slice<NBK, P>, P::bytes);
            if (e != cudaSuccess) return e;
            k_chi0_slice<NBK, P><<<g->nb, P::threads, P::bytes, st>>>(Grt, g->tw_k, g->n8, g->nw0, chirt, chiq);
            return launched();
        });
    }
};
template <int NBK>
struct RunVertexQ {
    static cudaError_t run(const GridDev *g, const double *chiq, double *Vr, double U, const double *Usc, double T,
                           cudaStream_t st) {
        const double normFact = T / ((double)g->nk0 * g->nk0);
        return with_plan<NBK, SlicePlan<NBK>, 1>(g->nb, [&](auto plan) {
            using P = decltype(plan);
            cudaError_t e = set_smem(k_vertex_q<NBK, P>, P::bytes);
            if (e != cudaSuccess) return e;
            k_vertex_q<NBK, P><<<g->nb, P::threads, P::bytes, st>>>(chiq, g->tw_k, g->n8, g->nb, normFact, U, Usc, Vr);
            return launched();
        });
    }
};
template <int NBK>
struct RunSigmaBoundary {
    template <class GT>
    static cudaError_t run(const GridDev *g, const GT *Grt, const double *V, const double *dchirt0,
                           const double *dG0p, double mu0, double U, const double *Usc, double *dS, const Bp *b,
                           cudaStream_t st) {
        const size_t smw = SliceSmem<NBK, SliceGroups<NBK>::wide>::bytes;
        cudaError_t e = set_smem(k_sigma_boundary<NBK, GT>, smw);
        if (e != cudaSuccess) return e;
        k_sigma_boundary<NBK, GT><<<dim3(2, 1, b->P), kSliceThreads, smw, st>>>(g->er, g->tw_k, Grt, V, dchirt0, dG0p,
                                                                                g->n8, g->nw0, g->n8p, mu0, U, Usc, dS,
                                                                                *b);
        return launched();
    }
};
template <int NBK>
struct RunSigmaSlice {
    static cudaError_t run(const GridDev *g, const double *Grt, const double *V, double *sigt, cudaStream_t st) {
        return with_plan<NBK, SlicePlan<NBK>, 1>(g->nw0 + 1, [&](auto plan) {
            using P = decltype(plan);
            cudaError_t e = set_smem(k_sigma_slice<NBK, P>, P::bytes);
            if (e != cudaSuccess) return e;
            const int ahead = resident_ctas(k_sigma_slice<NBK, P>, P::threads, P::bytes);
            k_sigma_slice<NBK, P><<<g->nw0 + 1, P::threads, P::bytes, st>>>(Grt, V, g->tw_k, g->n8, g->nw0, ahead, sigt);
            return launched();
        });
    }
};

template <int N>
dim3 tau3_grid(const GridDev &g, const Bp &b) {
    return dim3((g.n8p / 2 + Tau3Plan<N>::pairs - 1) / Tau3Plan<N>::pairs, 1, b.P);
}
// more column pairs than one wave of the pair kernels (256 threads, two CTAs an SM) takes
inline bool tau_groups(const GridDev &g, const Bp &b) {
    return (long long)(g.n8p / 2) * b.P > 2LL * sm_count();
}
template <int N>
struct RunChi0Tau {
    // (a batched launch, b->pp set, has no four-column tiling: the default instead)
    static cudaError_t run(const GridDev *g, double *chiq, const double *dchiqt0, double *cinf, double *cinf2,
                           double T, bool keep, const Bp *b, cudaStream_t st) {
        cudaError_t e;
        const int tile = tau_tile(keep ? kTauChi0Keep : kTauChi0, N);
        if constexpr (N <= kTau3Max) {
            if (!keep && (tile == 0 || (tile == 1 && b->pp)) && tau_groups(*g, *b)) {
                const size_t sm = Tau3Plan<N>::bytes;
                if ((e = set_smem(k_chi0_tau3<N>, sm)) != cudaSuccess) return e;
                k_chi0_tau3<N><<<tau3_grid<N>(*g, *b), Tau3Plan<N>::threads, sm, st>>>(
                    chiq, dchiqt0, cinf, cinf2, g->spl_half, g->tw_w, T, g->n8, g->n8p, *b);
                return launched();
            }
        }
        if constexpr (N / 8 <= 256) {
            if (tile == 2) {
                const size_t sm = Tau2Smem<N>::bytes;
                if ((e = set_smem(k_chi0_tau2<N, 8>, sm)) != cudaSuccess) return e;
                k_chi0_tau2<N, 8><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(chiq, dchiqt0, cinf, cinf2,
                                                                             g->spl_half, g->tw_w, T, g->n8, *b);
                return launched();
            }
        }
        if constexpr (N / 16 <= 256) {
            if (tile != 1 || b->pp) {
                const size_t sm = Tau2Smem<N>::bytes;
                if ((e = set_smem(k_chi0_tau2<N>, sm)) != cudaSuccess) return e;
                k_chi0_tau2<N><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(chiq, dchiqt0, cinf, cinf2, g->spl_half,
                                                                          g->tw_w, T, g->n8, *b);
                return launched();
            }
        }
        const size_t sm = TauSmem<N>::bytes(N / 2 + 1);
        e = set_smem(k_chi0_tau<N>, sm);
        if (e != cudaSuccess) return e;
        k_chi0_tau<N><<<g->n8p / 4, TauSmem<N>::threads, sm, st>>>(chiq, dchiqt0, cinf, cinf2, g->spl_half, g->tw_w,
                                                                    T, g->n8);
        return launched();
    }
};
template <int N>
struct RunVertexTau {
    static cudaError_t run(const GridDev *g, double *Vr, const double *chirt, double U, const double *Usc,
                           const Bp *b, cudaStream_t st) {
        cudaError_t e;
        const int tile = tau_tile(kTauVertex, N);
        if constexpr (N / 8 <= 256) {
            if (tile == 2) {
                const size_t sm = Tau2Smem<N>::bytes;
                if ((e = set_smem(k_vertex_tau2<N, 8>, sm)) != cudaSuccess) return e;
                k_vertex_tau2<N, 8><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(Vr, chirt, g->tw_w, U, Usc, g->n8,
                                                                               *b);
                return launched();
            }
        }
        if constexpr (N <= kTau3Max) {
            if ((tile != 1 || b->pp) && tau_groups(*g, *b)) {
                const size_t sm = Tau3Plan<N>::bytes;
                if ((e = set_smem(k_vertex_tau3<N>, sm)) != cudaSuccess) return e;
                k_vertex_tau3<N><<<tau3_grid<N>(*g, *b), Tau3Plan<N>::threads, sm, st>>>(Vr, chirt, g->tw_w, U, Usc, g->n8,
                                                                                          g->n8p, *b);
                return launched();
            }
        }
        if (tile != 1 || b->pp) {
            const size_t sm = Tau2Smem<N>::bytes;
            if ((e = set_smem(k_vertex_tau2<N>, sm)) != cudaSuccess) return e;
            k_vertex_tau2<N><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(Vr, chirt, g->tw_w, U, Usc, g->n8, *b);
            return launched();
        }
        const size_t sm = TauSmem<N>::bytes(N / 2 + 1);
        e = set_smem(k_vertex_tau<N>, sm);
        if (e != cudaSuccess) return e;
        k_vertex_tau<N><<<g->n8p / 4, TauSmem<N>::threads, sm, st>>>(Vr, chirt, g->tw_w, U, Usc, g->n8);
        return launched();
    }
};
template <int N>
struct RunSigmaTau {
    static cudaError_t run(const GridDev *g, const double *sigt, const double *dS, double2 *S, double *s2, double *s3,
                           double *s4, double *sinf, double T, const Bp *b, cudaStream_t st) {
        cudaError_t e;
        const int tile = tau_tile(kTauSigma, N);
        if constexpr (N / 8 <= 256) {
            if (tile == 2) {
                const size_t sm = Tau2Smem<N>::bytes;
                if ((e = set_smem(k_sigma_tau2<N, 8>, sm)) != cudaSuccess) return e;
                k_sigma_tau2<N, 8><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(
                    sigt, dS, S, s2, s3, s4, sinf, g->spl_full, g->tw_w, g->ht_w, T, g->n8, g->n8p, *b);
                return launched();
            }
        }
        if constexpr (N <= kTau3Max) {
            if ((tile != 1 || b->pp) && tau_groups(*g, *b)) {
                const size_t sm = Tau3Plan<N>::bytes;
                if ((e = set_smem(k_sigma_tau3<N>, sm)) != cudaSuccess) return e;
                k_sigma_tau3<N><<<tau3_grid<N>(*g, *b), Tau3Plan<N>::threads, sm, st>>>(
                    sigt, dS, S, s2, s3, s4, sinf, g->spl_full, g->tw_w, g->ht_w, T, g->n8, g->n8p, *b);
                return launched();
            }
        }
        if (tile != 1 || b->pp) {
            const size_t sm = Tau2Smem<N>::bytes;
            if ((e = set_smem(k_sigma_tau2<N>, sm)) != cudaSuccess) return e;
            k_sigma_tau2<N><<<dim3(g->n8p / 2, 1, b->P), 256, sm, st>>>(sigt, dS, S, s2, s3, s4, sinf, g->spl_full,
                                                                       g->tw_w, g->ht_w, T, g->n8, g->n8p, *b);
            return launched();
        }
        const size_t sm = TauSmem<N>::bytes(N + 1);
        if ((e = set_smem(k_sigma_tau<N>, sm)) != cudaSuccess) return e;
        k_sigma_tau<N><<<g->n8p / 4, TauSmem<N>::threads, sm, st>>>(sigt, dS, S, s2, s3, s4, sinf, g->spl_full,
                                                                     g->tw_w, g->ht_w, T, g->n8, g->n8p);
        return launched();
    }
};

}  // namespace

long long launches_total() { return g_launches.load(); }
long long launches_thread() { return t_launches; }
void add_launches(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

cudaError_t smem_optin(const void *fn) {
    static std::mutex mu;
    static std::set<std::pair<const void *, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({fn, dev})) return cudaSuccess;
    int optin = 0;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, fn)) != cudaSuccess) return e;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e == cudaSuccess) done.insert({fn, dev});
    return e;
}

bool supported_grid(int nk0, int nw0) {
    const int nbk = nk0 / 2 + 1;
    const bool k_ok = nbk == 5 || nbk == 9 || nbk == 17 || nbk == 33 || nbk == 65 || nbk == 129;
    const bool w_ok = nw0 >= 16 && nw0 <= 4096 && (nw0 & (nw0 - 1)) == 0;
    return k_ok && w_ok && nk0 == 2 * (nbk - 1);
}

cudaError_t launch_gslice(const GridDev &g, double *Grt, double mu0, double T, cudaStream_t st) {
    return dispatch_nbk<RunGslice>(g.nbk, &g, Grt, mu0, T, st);
}

cudaError_t launch_chi0_boundary(const GridDev &g, const double *Grt, double mu0, double T, double *dG0p,
                                 double *dtau_chirt0, double *dtau_chiqt0, cudaStream_t st) {
    const Bp b;
    return dispatch_nbk<RunChi0Boundary>(g.nbk, &g, Grt, mu0, T, dG0p, dtau_chirt0, dtau_chiqt0, &b, st);
}
cudaError_t launch_chi0_boundary(const GridDev &g, const float *Grt, double mu0, double T, double *dG0p,
                                 double *dtau_chirt0, double *dtau_chiqt0, cudaStream_t st, const Bp &b) {
    return dispatch_nbk<RunChi0Boundary>(g.nbk, &g, Grt, mu0, T, dG0p, dtau_chirt0, dtau_chiqt0, &b, st);
}

// eps_k on the octant (hamiltonien::calc_ek, src/hamiltonien.cpp:358-375), rounded
// operation by operation as the host expression is, the hopping table and the tail
// power sums.  The host's loops and copies of these tables cost 15 to 60 us a model,
// and a batch's 64 points were tabulated one by one before their group could start.
__global__ void __launch_bounds__(256)
    k_model_tables(const double *__restrict__ ktab, int nbk, int n8, const ModelTables m, double *__restrict__ ek,
                   double *__restrict__ er, double *__restrict__ tailq, double *__restrict__ tailP, Bp b) {
    ek = at(ek, b.arena);
    er = at(er, b.arena);
    const double tp = bpar(b, kPpTp, m.tp), tpp = bpar(b, kPpTpp, m.tpp), t3 = bpar(b, kPpT3, m.t3);
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (!b.pp) {
        if (o < kTailQ) tailq[o] = m.tailq[o];
        if (o < kTailP) tailP[o] = m.tailP[o];
    }
    if (o >= n8) return;
    int l, q;
    oct_lm(o, l, q);
    const Rn cl(ktab[l]), cm(ktab[q]), dl(ktab[2 * nbk + l]), dm(ktab[2 * nbk + q]);
    ek[o] = (Rn(-2.0) * (cl + cm) - Rn(4.0) * Rn(tp) * cl * cm - Rn(2.0) * Rn(tpp) * (dl + dm) -
             Rn(4.0) * Rn(t3) * (dl * cm + dm * cl)).v;
    er[o] = o == 1 ? -1.0 : o == 2 ? -tp : o == 3 ? -tpp : o == 4 ? -t3 : 0.0;
}
cudaError_t launch_model_tables(const GridDev &g, const ModelTables &m, cudaStream_t st, const Bp &b) {
    k_model_tables<<<dim3((g.n8 + 255) / 256, 1, b.P), 256, 0, st>>>(g.ktab, g.nbk, g.n8, m, g.ek, g.er, g.tailq,
                                                                      g.tailP, b);
    return launched();
}

cudaError_t launch_gk_table(const GridDev &g, double mu0, double T, cudaStream_t st, const Bp &b) {
    k_gk_table<<<dim3((g.n8 + 255) / 256, 1, b.P), 256, 0, st>>>(g.ek, g.n8, mu0, T, (double)g.nk0 * g.nk0, g.gk, b);
    return launched();
}

cudaError_t launch_chi0_slice(const GridDev &g, const double *Grt, double *chirt, double *chiq, cudaStream_t st) {
    return dispatch_nbk<RunChi0Slice>(g.nbk, &g, Grt, chirt, chiq, st);
}

cudaError_t launch_chi0_tau(const GridDev &g, double *chiq, const double *dtau_chiqt0, double *chi0_inf,
                            double *chi0_inf2, double T, cudaStream_t st, bool keep, const Bp &b) {
    return dispatch_nw<RunChi0Tau>(g.nw0, &g, chiq, dtau_chiqt0, chi0_inf, chi0_inf2, T, keep, &b, st);
}

cudaError_t launch_sumrule(const GridDev &g, const double *chiq, const double *chi0_inf, const double *chi0_inf2,
                           double Uv, double sign, double T, Reduce r, cudaStream_t st, int jdir, int tail) {
    const double Nq = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    if (jdir < 0 || jdir > g.nb) jdir = g.nb;
    const int nblk = g.n8p / 4;
    if (jdir < g.nb && !tail) {
        // low frequencies only: a short grid over the flattened (block, j) index
        const int grid = (int)std::min<long long>(std::max(1, 2 * sm_count()), ((long long)nblk * jdir + kRedThreads - 1) / kRedThreads);
        k_sumrule_low<<<std::max(grid, 1), kRedThreads, 0, st>>>(reinterpret_cast<const double4 *>(chiq), g.w16,
                                                                  g.nb, nblk, jdir, Uv, sign, T / Nq, r);
        return launched();
    }
    k_sumrule<<<nblk, kRedThreads, 0, st>>>(reinterpret_cast<const double4 *>(chiq), chi0_inf, chi0_inf2, g.w16,
                                            g.tailq, g.nb, jdir, tail, Uv, sign, T, T / Nq, r);
    return launched();
}

cudaError_t launch_sumrule_tan(const GridDev &g, const double *chiq, const double *dchiq, const double *chi0_inf,
                               const double *chi0_inf2, const double *dchi0_inf, const double *dchi0_inf2, double Usp,
                               double Uch, double T, Reduce r, cudaStream_t st) {
    const double Nq = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_sumrule_tan<<<g.n8p / 4, kRedThreads, 0, st>>>(reinterpret_cast<const double4 *>(chiq),
                                                     reinterpret_cast<const double4 *>(dchiq), chi0_inf, chi0_inf2,
                                                     dchi0_inf, dchi0_inf2, g.w16, g.nb, Usp, Uch, T, T / Nq, r);
    return launched();
}

cudaError_t launch_tail_moments(const GridDev &g, const double *chi0_inf, const double *chi0_inf2, double T,
                                Reduce r, cudaStream_t st, const Bp &b) {
    constexpr int NV = kMomP + 1;
    const int nblk = grid_for(g.n8, 256);
    k_tail_moments<<<dim3(nblk, 1, b.P), 256, 0, st>>>(chi0_inf, chi0_inf2, g.w16, g.tailq, g.n8, g.nb, T, r.partial,
                                                        b);
    cudaError_t e = launched();
    if (e != cudaSuccess) return e;
    e = finish<NV>(r, nblk, 0.0, st, b);
    if (e != cudaSuccess) return e;
    // the per-block maxima -> result[NV]
    k_max_finish<<<dim3(1, 1, b.P), 32, 0, st>>>(r.partial + (2 * kMomP + 1) * kMaxBlocks, nblk, r.result + NV, b);
    return launched();
}

namespace {

// double-double value hi + lo, |lo| <= ulp(hi) / 2
struct DD {
    double hi, lo;
};
__device__ __forceinline__ DD dd_add(DD a, DD b) {
    double s, e;
    two_sum(a.hi, b.hi, s, e);
    e += a.lo + b.lo;
    const double h = s + e;
    return DD{h, e - (h - s)};
}
__device__ __forceinline__ DD dd_shfl_down(DD a, int off) {
    return DD{__shfl_down_sync(0xffffffffu, a.hi, off), __shfl_down_sync(0xffffffffu, a.lo, off)};
}

// Block k < kMomP: suffix sums of moment k over the frequencies; block
// kMomP: suffix maxima of cmax and the tail values.  Each thread takes a
// chunk of consecutive frequencies; the chunk totals are combined by a warp
// suffix scan and the warps' totals in a fixed order, so the sums are
// deterministic.
__global__ void __launch_bounds__(256)
    k_moment_suffix(const double *__restrict__ mom, const double *__restrict__ cmax, const double *__restrict__ tail,
                    int nb, double *__restrict__ mom_suf, double *__restrict__ cmax_suf, double *__restrict__ tailm,
                    Bp b) {
    mom = at(mom, b.arena);
    cmax = at(cmax, b.arena);
    tail = at(tail, b.arena);
    mom_suf = at(mom_suf, b.arena);
    cmax_suf = at(cmax_suf, b.arena);
    tailm = at(tailm, b.arena);
    extern __shared__ double col[];
    __shared__ DD wtot[32];
    const int k = blockIdx.x;
    const bool is_max = k == kMomP;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) col[j] = is_max ? cmax[j] : mom[(size_t)j * kMomP + k];
    __syncthreads();
    const int C = (nb + blockDim.x - 1) / blockDim.x;
    const int s = min((int)threadIdx.x * C, nb), e = min(s + C, nb);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (is_max) {
        double m = 0.0;
        for (int j = e - 1; j >= s; --j) m = fmax(m, col[j]);
        for (int off = 1; off < 32; off <<= 1) {
            const double t = __shfl_down_sync(0xffffffffu, m, off);
            if (lane + off < 32) m = fmax(m, t);
        }
        if (lane == 0) wtot[warp].hi = m;
        double ex = __shfl_down_sync(0xffffffffu, m, 1);
        __syncthreads();
        if (lane == 31) ex = 0.0;
        for (int w = warp + 1; w < nw; ++w) ex = fmax(ex, wtot[w].hi);
        for (int j = e - 1; j >= s; --j) {
            ex = fmax(ex, col[j]);
            cmax_suf[j] = ex;
        }
        if (threadIdx.x == 0) {
            cmax_suf[nb] = 0.0;
            for (int i = 0; i < kMomP; ++i) tailm[i] = tail[i];
            tailm[kMomP] = tail[kMomP + 1];
        }
    } else {
        DD c{0.0, 0.0};
        for (int j = e - 1; j >= s; --j) c = dd_add(c, DD{col[j], 0.0});
        for (int off = 1; off < 32; off <<= 1) {
            const DD t = dd_shfl_down(c, off);
            if (lane + off < 32) c = dd_add(c, t);
        }
        if (lane == 0) wtot[warp] = c;
        DD ex = dd_shfl_down(c, 1);
        __syncthreads();
        if (lane == 31) ex = DD{0.0, 0.0};
        DD above{0.0, 0.0};
        for (int w = nw - 1; w > warp; --w) above = dd_add(above, wtot[w]);
        ex = dd_add(ex, above);
        for (int j = e - 1; j >= s; --j) {
            ex = dd_add(ex, DD{col[j], 0.0});
            mom_suf[(size_t)j * kMomP + k] = ex.hi + ex.lo;
        }
        if (threadIdx.x == 0) mom_suf[(size_t)nb * kMomP + k] = 0.0;
    }
}

}  // namespace

cudaError_t launch_moment_suffix(const GridDev &g, const double *mom, const double *cmax, const double *tail_result,
                                 double *mom_suf, double *cmax_suf, double *tailm, cudaStream_t st, const Bp &b) {
    const size_t sm = (size_t)g.nb * sizeof(double);
    cudaError_t e = set_smem(k_moment_suffix, sm);
    if (e != cudaSuccess) return e;
    k_moment_suffix<<<dim3(kMomP + 1, 1, b.P), 256, sm, st>>>(mom, cmax, tail_result, g.nb, mom_suf, cmax_suf, tailm,
                                                               b);
    return launched();
}

cudaError_t launch_chi0_moments(const GridDev &g, const double *chiq, double *mom, double *cmax, cudaStream_t st,
                                const Bp &b) {
    k_chi0_moments<<<dim3(g.nb, 1, b.P), 256, 0, st>>>(reinterpret_cast<const double4 *>(chiq), g.w16, g.nb,
                                                        g.n8p / 4, mom, cmax, b);
    return launched();
}

cudaError_t launch_trace_chi0(const GridDev &g, const double *chiq, const double *chi0_inf, const double *chi0_inf2,
                              double T, Reduce r, cudaStream_t st) {
    const double Nq = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_trace_chi0<<<g.n8p / 4, kRedThreads, 0, st>>>(reinterpret_cast<const double4 *>(chiq), chi0_inf, chi0_inf2,
                                                     g.w16, g.nb, T, Nq, r);
    return launched();
}

cudaError_t launch_vertex_q(const GridDev &g, const double *chiq, double *Vr, double U, const double *Usc, double T,
                            cudaStream_t st) {
    return dispatch_nbk<RunVertexQ>(g.nbk, &g, chiq, Vr, U, Usc, T, st);
}

cudaError_t launch_vertex_tau(const GridDev &g, double *Vr, const double *chirt, double U, const double *Usc,
                              cudaStream_t st, const Bp &b) {
    return dispatch_nw<RunVertexTau>(g.nw0, &g, Vr, chirt, U, Usc, &b, st);
}

cudaError_t launch_sigma_boundary(const GridDev &g, const double *Grt, const double *V, const double *dtau_chirt0,
                                  const double *dG0p, double mu0, double U, const double *Usc, double *dS,
                                  cudaStream_t st) {
    const Bp b;
    return dispatch_nbk<RunSigmaBoundary>(g.nbk, &g, Grt, V, dtau_chirt0, dG0p, mu0, U, Usc, dS, &b, st);
}
cudaError_t launch_sigma_boundary(const GridDev &g, const float *Grt, const double *V, const double *dtau_chirt0,
                                  const double *dG0p, double mu0, double U, const double *Usc, double *dS,
                                  cudaStream_t st, const Bp &b) {
    return dispatch_nbk<RunSigmaBoundary>(g.nbk, &g, Grt, V, dtau_chirt0, dG0p, mu0, U, Usc, dS, &b, st);
}

cudaError_t launch_sigma_slice(const GridDev &g, const double *Grt, const double *V, double *sigt, cudaStream_t st) {
    return dispatch_nbk<RunSigmaSlice>(g.nbk, &g, Grt, V, sigt, st);
}

cudaError_t launch_sigma_tau(const GridDev &g, const double *sigt, const double *dS, double2 *S, double *s2,
                             double *s3, double *s4, double *sinf, double T, cudaStream_t st, const Bp &b) {
    return dispatch_nw<RunSigmaTau>(g.nw0, &g, sigt, dS, S, s2, s3, s4, sinf, T, &b, st);
}

cudaError_t launch_trace_diff_G(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                const double *s4, const double *sinf, double mu0, double pmu, double T, Reduce r,
                                cudaStream_t st, int jdir) {
    const int NO = g.nw0 / 2;
    const int tail = (jdir < 0) ? 1 : 0;
    if (jdir < 0 || jdir > NO) jdir = NO;
    const int nblk = g.n8p / 4;
    if (!tail) {
        const int grid = (int)std::min<long long>(std::max(1, 2 * sm_count()), ((long long)nblk * jdir + kRedThreads - 1) / kRedThreads);
        k_trace_diff_G_low<<<std::max(grid, 1), kRedThreads, 0, st>>>(S, s2, s3, sinf, g.ek, g.w16, g.nw0, nblk, mu0,
                                                                       pmu, T, jdir, r);
        return launched();
    }
    k_trace_diff_G<true><<<nblk, kRedThreads, 0, st>>>(S, s2, s3, s4, sinf, g.ek, g.w16, g.nw0, mu0, pmu, T, jdir, tail,
                                                  r);
    return launched();
}

cudaError_t launch_trace_value_G(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                 const double *s4, const double *sinf, double mu0, double pmu, double T, Reduce r,
                                 cudaStream_t st) {
    k_trace_diff_G<false><<<g.n8p / 4, kRedThreads, 0, st>>>(S, s2, s3, s4, sinf, g.ek, g.w16, g.nw0, mu0, pmu, T,
                                                             g.nw0 / 2, 1, r);
    return launched();
}

cudaError_t launch_trace_self_G(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                const double *sinf, double mu0, double T, Reduce r, cudaStream_t st) {
    const double nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_trace_self_G<<<g.n8p / 4, kRedThreads, 0, st>>>(S, s2, s3, sinf, g.ek, g.w16, g.nw0, mu0, T, nk02, r);
    return launched();
}

cudaError_t launch_trace_self_G2(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                 const double *sinf, double mu, double T, Reduce r, cudaStream_t st) {
    const double nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_trace_self_G2<<<g.n8p / 4, kRedThreads, 0, st>>>(S, s2, s3, sinf, g.ek, g.w16, g.nw0, mu, T, nk02, r);
    return launched();
}

bool zero_by_host(const GridDev &g, int max_blocks) {
    return max_blocks > 0 && 2 * max_blocks < sm_count() && g.n8p / 4 > 4 * max_blocks;
}

cudaError_t launch_pade_sigma(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                              const double *sinf, const int *nidx, int Nn, const double2 *z, int Nz, int mode,
                              double mu, double T, double2 *out_sig, double *out_A, cudaStream_t st) {
    if (Nn < 2 || Nn > kPadeMax || Nn > g.nw0 / 2) return cudaErrorInvalidValue;
    k_pade_sigma<<<g.n8, 128, 0, st>>>(S, s2, s3, sinf, g.ek, nidx, Nn, z, Nz, mode, g.n8, g.nw0, mu, T,
                                                      out_sig, out_A);
    return launched();
}

cudaError_t launch_gwn_local(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                             const double *sinf, double mu, double T, double2 *out, cudaStream_t st) {
    const double nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_gwn_local<<<g.nw0 / 2, 256, 0, st>>>(S, s2, s3, sinf, g.ek, g.w16, g.n8, g.nw0, mu, T, nk02, out);
    return launched();
}

cudaError_t launch_mu0_newton(const GridDev &g, double n, double T, Reduce r, cudaStream_t st, const Bp &b) {
    k_mu0_newton<<<dim3(1, 1, b.P), 1024, 0, st>>>(g.ek, g.n8, g.nbk, n, T, 4.0 * (g.nbk - 1) * (g.nbk - 1),
                                                    r.result, b);
    return launched();
}

cudaError_t launch_chi0max(const GridDev &g, const double *chiq, Reduce r, cudaStream_t st, const Bp &b) {
    k_chi0max<<<dim3(1, 1, b.P), 1024, 0, st>>>(chiq, g.n8, g.nb, r.result, b);
    return launched();
}

cudaError_t launch_unblock(const double *src, double *dst, int NJ, int nrows, int n8, cudaStream_t st) {
    const int nb = grid_for((long long)nrows * n8, 256);
    k_unblock<<<nb, 256, 0, st>>>(src, dst, NJ, nrows, n8);
    return launched();
}

cudaError_t launch_unblock_c(const double2 *src, double2 *dst, int NJ, int nrows, int n8, cudaStream_t st) {
    const int nb = grid_for((long long)nrows * n8, 256);
    k_unblock_c<<<nb, 256, 0, st>>>(src, dst, NJ, nrows, n8);
    return launched();
}

cudaError_t launch_sigma_full32(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                const double *sinf, double T, float2 *dst, cudaStream_t st) {
    const int NO = g.nw0 / 2;
    const int nb = grid_for((long long)NO * g.n8, 256);
    k_sigma_full32<<<nb, 256, 0, st>>>(S, s2, s3, sinf, NO, g.n8, T, dst);
    return launched();
}

cudaError_t launch_block(const double *src, double *dst, int NJ, int nrows, int n8, cudaStream_t st) {
    const int nb = grid_for((long long)nrows * n8, 256);
    k_block<<<nb, 256, 0, st>>>(src, dst, NJ, nrows, n8);
    return launched();
}

cudaError_t launch_block_c(const double2 *src, double2 *dst, int NJ, int nrows, int n8, cudaStream_t st) {
    const int nb = grid_for((long long)nrows * n8, 256);
    k_block_c<<<nb, 256, 0, st>>>(src, dst, NJ, nrows, n8);
    return launched();
}

cudaError_t launch_take_row(const double *src, int NJ, int j, int n8, double *dst, cudaStream_t st) {
    k_take_row<<<grid_for(n8, 256), 256, 0, st>>>(src, NJ, j, n8, dst);
    return launched();
}

cudaError_t launch_gather(const GatherPieces &p, unsigned *dst, int blocks, cudaStream_t st) {
    k_gather<<<blocks, 256, 0, st>>>(p, dst);
    return launched();
}

cudaError_t launch_store(double *dst, const double *v, int n, cudaStream_t st) {
    if (n < 0 || n > 4) return cudaErrorInvalidValue;
    StoreVals s;
    for (int i = 0; i < 4; ++i) s.v[i] = i < n ? v[i] : 0.0;
    s.n = n;
    k_store<<<1, 32, 0, st>>>(s, dst);
    return launched();
}

}  // namespace tpsc
