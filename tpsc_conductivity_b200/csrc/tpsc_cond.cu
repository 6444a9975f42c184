// tpsc_cond.cu -- current-current correlator chi_jj(iqn) with the
// Maki-Thompson vertex correction, and the diamagnetic term kx0, in FP64
// (cond_opt::calc_chijj_vertex_corr_all_optim, bubble + Maki-Thompson branch,
// src/cond_opt.cpp:2537-4286).
//
// The reference works on the K4 grid of interior kx points: l = 0..nbk-3
// stands for kx = (l+1) pi/(nbk-1), m = 0..nbk-1 for ky = m pi/(nbk-1); the
// current vertex d eps/d kx is odd in kx and even in ky, so the real-space
// transforms are DST-I (RODFT00) along kx and DCT-I (REDFT00) along ky.
// Three kernel families:
//  * cond slices: one CTA per (tau_j, h or f0).  h(r, tau) and f0(r, tau)
//    are built from eps_k, transformed, multiplied by 2 V(r, tau) and
//    transformed back (src/cond_opt.cpp:2696-2908, 3027-3112), in shared
//    memory; the result is written in a two-column-block layout (the two
//    columns of a pair contiguous along tau) for the tau kernel.
//  * cond boundary: four CTAs for the tau-derivative end conditions of the
//    two splines (src/cond_opt.cpp:2744-2887, 2910-3025).
//  * cond tau: a persistent kernel looping over pairs of K4
//    columns.  Per pair: the two splines + pre-twiddled FFTs give
//    J(k, ikn) and J0(k, ikn); G(k, ikn) = T/(ikn - eps + mu - Sigma) with
//    its analytic tail; the two back-transforms to tau; the spline + FFT of
//    G J (Maki-Thompson moment) and of -G(tau) G(beta - tau) (bubble)
//    (src/cond_opt.cpp:3179-3849).  Sigma is read once per column.  Every
//    CTA accumulates its columns' contributions in its own row of a partial
//    array; a finish kernel adds the rows in a fixed order.
// Plus the kx = 0, pi line sums of kx0 (src/cond_opt.cpp:3993-4173).
#include <cuda_runtime.h>
#include <stdint.h>

#include "tpsc_device.cuh"

namespace tpsc {

namespace {


__device__ __forceinline__ double cabs2(double2 z) { return hypot(z.x, z.y); }

// principal square root
__device__ __forceinline__ double2 csqrt2(double2 z) {
    const double r = cabs2(z);
    if (r == 0.0) return make_double2(0.0, z.y);
    const double t = sqrt(0.5 * (r + fabs(z.x)));
    if (z.x >= 0.0) return make_double2(t, z.y / (2.0 * t));
    return make_double2(fabs(z.y) / (2.0 * t), copysign(t, z.y));
}


// z^2 + B z + C at x and its derivative
__device__ __forceinline__ void quad_eval(double2 x, double2 B, double2 C, double2 &y, double2 &p) {
    y = cadd(cadd(cmul(x, x), cmul(B, x)), C);
    p = cadd(cscale(x, 2.0), B);
}

// Roots of z^2 + B z + C: closed form, then Newton polish (tolerance 1e-16 on
// |p(x)|, at most 10 steps, halving back when a step makes |p| grow), a
// polished root kept only if it improved |p| (generique::find_roots_2pol,
// src/generique.cpp:1666-1727, with A = 1).  Real coefficients with two real
// roots need no polish: the root that adds the magnitudes of -B and the square
// root is exact to an ulp, the other is C over it (the chain of hypots and
// complex divisions of ten steps made the tau kernel's column constants 27 us).
__device__ void roots_2pol(double2 B, double2 C, double2 &r0, double2 &r1) {
    const double disc = fma(B.x, B.x, -4.0 * C.x);
    if (B.y == 0.0 && C.y == 0.0 && C.x != 0.0 && disc > 0.0) {
        const double R = sqrt(disc);
        const double big = -0.5 * (B.x + (B.x >= 0.0 ? R : -R)), small = C.x / big;
        r0 = make_double2(B.x >= 0.0 ? big : small, 0.0);
        r1 = make_double2(B.x >= 0.0 ? small : big, 0.0);
        return;
    }
    const double2 R = csqrt2(csub(cmul(B, B), cscale(C, 4.0)));
    double2 root[2] = {cscale(csub(make_double2(-B.x, -B.y), R), 0.5), cscale(cadd(make_double2(-B.x, -B.y), R), 0.5)};
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        double2 x = root[k], y, p;
        quad_eval(x, B, C, y, p);
        const double y0 = cabs2(y);
        for (int it = 0; it < 10 && cabs2(p) != 0.0 && cabs2(y) > 1.0e-16; ++it) {
            const double2 x2 = x;
            const double ay2 = cabs2(y);
            const double2 c = csub(y, cmul(p, x));
            x = cdiv(make_double2(-c.x, -c.y), p);
            quad_eval(x, B, C, y, p);
            if (ay2 < cabs2(y)) {
                x = cscale(cadd(x, x2), 0.5);
                quad_eval(x, B, C, y, p);
            }
        }
        if (cabs2(y) < y0) root[k] = x;
    }
    r0 = root[0];
    r1 = root[1];
}

// ---------------------------------------------------------------------------
// per-K4-point constants of the h and f0 slices (src/cond_opt.cpp:2696-2827):
// x = eps - mu0; with E(t) = exp(-x t) (x > 0) or exp(x (beta - t)) (x <= 0)
//   h(t)  = A E(t),  f0(t) = (A t + B) E(t)
//   x > 0:  A = dek/L^2 / (e^{-x/T} + 1),  B = -dek/L^2 e^{-x/T} / (T (e^{-x/T} + 1)^2)
//   x <= 0: A = dek/L^2 / (e^{x/T} + 1),   B = -dek/L^2 / (T (e^{x/T} + 1)^2)
// tab[4c..4c+2] = (x, A, B)
// ---------------------------------------------------------------------------
// d eps/d kx and d2 eps/d kx2 (hamiltonien::grad_ek direction 0 and Hessian_ek
// (0, 0), src/hamiltonien.cpp:134-155) on k = (l+1, m) pi/(nbk-1)
// (src/cond_opt.cpp:2588-2611), and the second on the kx = 0, pi lines, from the
// grid's table of sines and cosines.  Ten host sines and cosines a point took 0.3 ms at
// 128 x 128 and 1.2 ms at 256 x 256 of every call.
__global__ void __launch_bounds__(256)
    k_cond_model(const double *__restrict__ ktab, int nbk, int K4, double tp, double tpp, double t3,
                 double *__restrict__ dek, double *__restrict__ d2ek, double *__restrict__ d2line) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K4 + 2 * nbk) return;
    const int line = i - K4;  // >= 0: the points of the two lines
    const int l = line < 0 ? i / nbk + 1 : (line < nbk ? 0 : nbk - 1), m = (line < 0 ? i : line) % nbk;
    const double *c1 = ktab, *s1 = ktab + nbk, *c2 = ktab + 2 * nbk, *s2 = ktab + 3 * nbk;
    const double h = 2.0 * c1[l] + 4.0 * tp * c1[l] * c1[m] + 8.0 * tpp * c2[l] +
                     4.0 * t3 * (4.0 * c2[l] * c1[m] + c2[m] * c1[l]);
    if (line >= 0) {
        d2line[line] = h;
        return;
    }
    d2ek[i] = h;
    dek[i] = 2.0 * s1[l] + 4.0 * tp * s1[l] * c1[m] + 4.0 * tpp * s2[l] +
             4.0 * t3 * (2.0 * s2[l] * c1[m] + c2[m] * s1[l]);
}

__global__ void k_cond_table(const double *__restrict__ ek, const double *__restrict__ dek, int K4, int nbk,
                             double mu0, double T, double nf, double *__restrict__ tab) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= K4) return;
    const int l = c / nbk, m = c % nbk;
    const double x = ek[oct_index(l + 1, m)] - mu0;
    const double d = nf * dek[c];
    double A, B;
    if (x > 0) {
        const double ep = exp(-x / T);
        A = d / (ep + 1.0);
        B = -d * ep / (T * (ep + 1.0) * (ep + 1.0));
    } else {
        const double en = exp(x / T);
        A = d / (en + 1.0);
        B = -d / (T * (en + 1.0) * (en + 1.0));
    }
    tab[4 * c] = x;
    tab[4 * c + 1] = A;
    tab[4 * c + 2] = B;
    tab[4 * c + 3] = 0.0;
}

// h V(r, tau_j) (blockIdx.y = 0) or f0 V(r, tau_j) (blockIdx.y = 1),
// j = blockIdx.x = 0..Nw0: the slice, its DST x DCT, times 2 V(r, tau_j)
// (V(r, beta - tau) for tau > beta/2; r = (l+1, m) folded into the octant),
// DST x DCT again.  The first transform at tau = 0 and beta is kept in
// `pre` for the boundary kernel.
template <int NBK>
__global__ void __launch_bounds__(SlicePlan<NBK>::threads, SlicePlan<NBK>::blocks)
    k_cond_slice(const double *__restrict__ tab, const double *__restrict__ V, const double2 *__restrict__ tw,
                 int nw0, double T, int K4p, double *__restrict__ hV, double *__restrict__ f0V,
                 double *__restrict__ pre) {
    constexpr int K4 = (NBK - 2) * NBK;
    extern __shared__ __align__(16) double S[];
    const auto *tws = plan_twiddles<NBK>(S, tw);
    const int j = blockIdx.x, y = blockIdx.y;
    const int nb = nw0 / 2 + 1;
    const double t = j / (nw0 * T);
    const double bt = 1.0 / T - t;
    batched<4>(
        K4,
        [&](int c) -> double3 {
            const double2 xa = *reinterpret_cast<const double2 *>(tab + 4 * c);
            return make_double3(xa.x, xa.y, y == 0 ? 0.0 : tab[4 * c + 2]);
        },
        [&](int c, double3 v) {
            const double E = exp(v.x > 0 ? -v.x * t : v.x * bt);
            S[c] = (y == 0) ? v.y * E : (v.y * t + v.z) * E;  // row l, column m: c = l NBK + m
        });
    __syncthreads();
    plan_dst_dct<NBK>(S, tws);
    const int jv = j < nb ? j : nw0 - j;
    const bool edge = (j == 0 || j == nw0);
    double *pe = pre + (size_t)(2 * y + (j == nw0 ? 1 : 0)) * K4p;
    batched<8>(
        K4, [&](int c) -> double { return V[bidx(jv, oct_index(c / NBK + 1, c % NBK), nb)]; },
        [&](int c, double w) {
            const double v = S[c];
            if (edge) pe[c] = v;
            S[c] = v * (2.0 * w);
        });
    __syncthreads();
    plan_dst_dct<NBK>(S, tws);
    double *out = (y == 0) ? hV : f0V;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) out[bidx2(j, c, nw0 + 1)] = S[c];
}

// End conditions of the two splines (src/cond_opt.cpp:2744-2887, 2910-3025):
// kind 0: dhV(0), 1: dhV(beta), 2: df0V(0), 3: df0V(beta) =
//   DST x DCT[ 2 D V(r, 0) +- P fact d/dtau chi0(r, 0) ]
// with D the transformed tau-derivative of h (f0) at the end, P the
// transformed h (f0) there, + at tau = 0 and - at beta.
template <int NBK>
__global__ void __launch_bounds__(kSliceThreads, 1)
    k_cond_boundary(const double *__restrict__ ek, const double *__restrict__ dek, const double *__restrict__ V,
                    const double *__restrict__ dchirt0, const double2 *__restrict__ tw, const double *__restrict__ pre,
                    int nw0, int K4p, double mu0, double T, double nf, double fact, double *__restrict__ dbound) {
    constexpr int K4 = (NBK - 2) * NBK;
    extern __shared__ __align__(16) double S[];
    const auto *tws = slice_twiddles<NBK, SliceGroups<NBK>::wide>(S, tw);
    const int kind = blockIdx.x;
    const int nb = nw0 / 2 + 1;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const int l = c / NBK, m = c % NBK;
        const double x = ek[oct_index(l + 1, m)] - mu0;
        const double d = nf * dek[c];
        double v;
        if (x > 0) {
            const double ep = exp(-x / T), q = ep + 1.0;
            switch (kind) {
                case 0: v = -d * x / q; break;
                case 1: v = -d * x * ep / q; break;
                case 2: v = d * (x * ep / (T * q * q) + 1.0 / q); break;
                default: v = d * ep * ((-x) * (1.0 / (T * q) - ep / (T * q * q)) + 1.0 / q); break;
            }
        } else {
            const double en = exp(x / T), q = en + 1.0;
            switch (kind) {
                case 0: v = -d * x * en / q; break;
                case 1: v = -d * x / q; break;
                case 2: v = d * en * (x / (T * q * q) + 1.0 / q); break;
                default: v = d * ((-x) * (1.0 / (T * q) - 1.0 / (T * q * q)) + 1.0 / q); break;
            }
        }
        S[c] = v;
    }
    __syncthreads();
    dst_dct_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    const double sg = (kind & 1) ? -1.0 : 1.0;
    const double *pe = pre + (size_t)kind * K4p;
    for (int c = threadIdx.x; c < K4; c += blockDim.x) {
        const int l = c / NBK, m = c % NBK;
        const int o = oct_index(l + 1, m);
        S[c] = 2.0 * S[c] * V[bidx(0, o, nb)] + sg * pe[c] * fact * dchirt0[o];
    }
    __syncthreads();
    dst_dct_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    for (int c = threadIdx.x; c < K4; c += blockDim.x) dbound[(size_t)kind * K4p + c] = S[c];
}

// ---------------------------------------------------------------------------
// the per-k tau kernel
// ---------------------------------------------------------------------------
// What the tau kernel takes per K4 column, from eps, mu and Sigma_inf alone:
// the roots r1, r2 of z^2 + (mu - eps) z - Sigma_inf, the prefactors of the
// analytic tails (src/cond_opt.cpp:3421-3467)
//   G0(tau) = -Re(u1 e1 + u2 e2),  Jinf(tau) = C1 Re(w1 j1 + w2 j2),
// and the tails' parts of k0, dG/dtau(0+, 0-) and (per C1) dJ/dtau(0, beta).
struct CondCol {
    double2 r1, r2, u1, u2, w1, w2;
    double k0, dGp, dGm, dJ0, dJb;
    double e, dk, d2, wt;
    int o, bin;
};
constexpr int kCondColWords = sizeof(CondCol) / sizeof(double);
static_assert(sizeof(CondCol) % sizeof(double) == 0, "copied by double words");

__global__ void __launch_bounds__(64)
    k_cond_cols(const double *__restrict__ ek, const double *__restrict__ dek, const double *__restrict__ d2ek,
                const int *__restrict__ bin, const double *__restrict__ sinfp, int K4, int K4p, int nbk, double mu,
                double T, CondCol *__restrict__ cols) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= K4p) return;
    const int cc = c < K4 ? c : K4 - 1;
    const int l = cc / nbk, m = cc % nbk;
    CondCol q;
    q.o = oct_index(l + 1, m);
    q.e = ek[q.o];
    q.dk = dek[cc];
    q.d2 = d2ek[cc];
    q.wt = c < K4 ? ((m == 0 || m == nbk - 1) ? 2.0 : 4.0) : 0.0;
    q.bin = bin ? bin[cc] : 0;
    double2 r1, r2;
    roots_2pol(make_double2(mu - q.e, 0.0), make_double2(-sinfp[0], 0.0), r1, r2);
    q.r1 = r1;
    q.r2 = r2;
    const double2 a1 = cdiv(r1, csub(r1, r2)), a2 = cdiv(r2, csub(r2, r1));
    const double2 b1 = cdiv(make_double2(1.0, 0.0), csub(r1, r2)), b2 = make_double2(-b1.x, -b1.y);
    auto branch = [&](double2 r, double2 av, double2 bv, double2 &u, double2 &w, double2 &fp, double2 &fm, double2 &fj,
                      double2 &fjb) {
        const bool big = r.x > 0;
        const double2 ex = big ? cexp2(cscale(r, -1.0 / T)) : cexp2(cscale(r, 1.0 / T));
        const double2 den = make_double2(ex.x + 1.0, ex.y), rb = cmul(r, bv);
        const double2 one = cdiv(av, den), exd = cdiv(cmul(av, ex), den);
        const double2 j1 = cdiv(rb, den), jx = cdiv(cmul(rb, ex), den);
        fp = big ? one : exd;
        fm = big ? exd : one;
        fj = big ? jx : j1;
        fjb = big ? j1 : jx;
        u = one;
        w = cdiv(bv, den);
    };
    double2 f1p, f1m, fj1, fj1b, f2p, f2m, fj2, fj2b;
    branch(r1, a1, b1, q.u1, q.w1, f1p, f1m, fj1, fj1b);
    branch(r2, a2, b2, q.u2, q.w2, f2p, f2m, fj2, fj2b);
    q.k0 = f1m.x + f2m.x;
    q.dGm = cmul(r1, f1m).x + cmul(r2, f2m).x;
    q.dGp = cmul(r1, f1p).x + cmul(r2, f2p).x;
    q.dJb = fj1b.x + fj2b.x;
    q.dJ0 = fj1.x + fj2.x;
    cols[c] = q;
}

// Two groups of G = N/16 threads, one per transform in flight, and as many CTAs
// per SM as leave 128 registers a thread
template <int N>
struct CondTauPlan {
    static constexpr int G = FftPlan<N>::G;
    static constexpr int threads = 2 * G < 32 ? 32 : 2 * G;
    static constexpr int blocks = 512 / threads > 12 ? 12 : 512 / threads;
    static constexpr int x_len = padded_len(N) + 2;        // N + 1 nodes
    static constexpr int n_hi = N / 64 + 1, n_lo = 64;     // two-level tails: tau_j, j = 64 hi + lo <= N
    static constexpr size_t tables_off = (size_t)2 * x_len * sizeof(double2);
    static constexpr size_t tails_off = tables_off + 2 * sizeof(TwoLevelTw);
    static constexpr size_t bytes = tails_off + (size_t)4 * (n_hi + n_lo) * sizeof(double);
};

struct CondTauArgs {
    const double2 *hV, *f0V;  // two-column blocks: the two columns of a pair as the parts of one complex
    const double *dbound;
    const double2 *S;
    const double *s2, *s3, *sinf;
    const CondCol *cols;
    const double *spl_full, *spl_half;
    const double2 *tw, *ht;
    double *partial;
    int K4, K4p, pw;
    double mu, T, nf;
};

// per-column values of the pair being processed
struct ColState {
    double2 v1, v2;                  // C1 w1, C1 w2
    double q0;                       // Re sum_n G^2 J0 / T, all n
    double k0, dGp, dGm, dJ0, dJb;
    double Gt0, Jt0, Jraw0;
    double dchi, integ;
    double CJ1b, CJ3b;
};

// analytic tails at tau: G0(tau) = Re(-u1 e1 - u2 e2), Jinf(tau) = Re(v1 j1 + v2 j2)
// (src/cond_opt.cpp:3574-3640)
__device__ __forceinline__ void tails(const CondCol &q, const ColState &s, double tau, double beta, double &g0,
                                      double &jinf) {
    const bool big1 = q.r1.x > 0, big2 = q.r2.x > 0;
    const double2 e1 = big1 ? cexp2(cscale(q.r1, -tau)) : cexp2(cscale(q.r1, beta - tau));
    const double2 j1 = big1 ? cexp2(cscale(q.r1, tau - beta)) : cexp2(cscale(q.r1, tau));
    const double2 e2 = big2 ? cexp2(cscale(q.r2, -tau)) : cexp2(cscale(q.r2, beta - tau));
    const double2 j2 = big2 ? cexp2(cscale(q.r2, tau - beta)) : cexp2(cscale(q.r2, tau));
    g0 = -cmul(q.u1, e1).x - cmul(q.u2, e2).x;
    jinf = cmul(s.v1, j1).x + cmul(s.v2, j2).x;
}

__device__ __forceinline__ double part_of(double2 z, int q) { return q == 0 ? z.x : z.y; }
// Persistent over column pairs; the pair's two real columns are the parts of one
// complex column throughout, in two buffers X1, X2 that two groups of threads
// spline and transform in place at the same time: f0 V beside h V, G beside J,
// the bubble beside the Maki-Thompson product.
// Bound: the FP64 pipe (six N-point FFTs, four splines) and the sweeps' and
// transforms' latencies at 16 warps per SM.  One transform at a time in 128 or
// 256 threads at 240 registers (8 warps per SM), with four exponentials, five
// more divisions per point and the roots' Newton polish in the pair loop took
// 8290 us at 256^2 x 4096 and 937 at 128^2 x 2048; this takes 3300 and 461.
// The tails' exponentials exp(-|r| tau_j) are products of two table entries
// (formed per pair) when the roots are real, as they are for Sigma_inf > 0.
template <int N>
__global__ void __launch_bounds__(CondTauPlan<N>::threads, CondTauPlan<N>::blocks) k_cond_tau(const CondTauArgs a) {
    using P = CondTauPlan<N>;
    constexpr int NJ = N + 1, NO = N / 2, NJ2 = NO + 1, G = P::G, NT = P::threads;
    extern __shared__ __align__(16) double2 X1[];
    double2 *X2 = X1 + P::x_len;
    TwoLevelTw *tw2 = reinterpret_cast<TwoLevelTw *>(reinterpret_cast<char *>(X1) + P::tables_off);
    const TwoLevelTw *ht2 = tw2 + 1;
    double *tails_hi = reinterpret_cast<double *>(reinterpret_cast<char *>(X1) + P::tails_off);
    double *tails_lo = tails_hi + 4 * P::n_hi;
    tau_tables(tw2, tw2 + 1, a.tw, a.ht, N);  // published by the first barrier of the pair loop
    __shared__ CondCol col[2];
    __shared__ ColState cs[2];
    __shared__ double2 d0s[2], dNs[2];            // end slopes of X1's and X2's columns
    __shared__ double2 sC1[2], sC2[2], sC3[2];    // tau moments of X1's and X2's columns
    __shared__ double sums[8], sV[2];
    const int tid = threadIdx.x, grp = tid / G, t = tid % G;
    double2 *const X = grp == 0 ? X1 : X2;
    const double T = a.T, h = 1.0 / (N * T), ih = 1.0 / h, beta = 1.0 / T, pT = kPi * T;
    const double sinf = a.sinf[0], mu = a.mu, nf = a.nf;
    constexpr int PWB = 2 * NJ2;
    double *part = a.partial + (size_t)blockIdx.x * a.pw;
    const int npairs = a.K4p / 2;

#pragma unroll 1
    for (int p = blockIdx.x; p < npairs; p += gridDim.x) {
        const int c0 = 2 * p;
        for (int j = tid; j < NJ; j += NT) {
            cp_async16(&X1[pidx(j)], a.f0V + (size_t)p * NJ + j);
            cp_async16(&X2[pidx(j)], a.hV + (size_t)p * NJ + j);
        }
        for (int i = tid; i < 2 * kCondColWords; i += NT)
            reinterpret_cast<double *>(col)[i] = reinterpret_cast<const double *>(a.cols + c0)[i];
        if (tid < 2) {
            // f0 V: rows 2, 3 of the end conditions; h V: rows 0, 1
            const double *b = a.dbound + (size_t)(tid == 0 ? 2 : 0) * a.K4p + c0;
            const bool two = c0 + 1 < a.K4;
            d0s[tid] = make_double2(b[0], two ? b[1] : 0.0);
            dNs[tid] = make_double2(b[a.K4p], two ? b[a.K4p + 1] : 0.0);
        }
        cp_async_wait_all();
        __syncthreads();
        const bool real_roots = col[0].r1.y == 0.0 && col[0].r2.y == 0.0 && col[1].r1.y == 0.0 && col[1].r2.y == 0.0;
        // exp(-|r| tau_j), column q and root k: row 2 q + k
        for (int i = tid; i < 4 * (P::n_hi + P::n_lo); i += NT) {
            const bool hi = i < 4 * P::n_hi;
            const int ii = hi ? i : i - 4 * P::n_hi, len = hi ? P::n_hi : P::n_lo, row = ii / len, e = ii % len;
            const CondCol &q = col[row >> 1];
            const double r = fabs((row & 1) ? q.r2.x : q.r1.x);
            (hi ? tails_hi : tails_lo)[ii] = exp(-r * ((hi ? 64 * e : e) * h));
        }
        // ---- f0 V and h V: splines and F = FFT_{+}[exp(i pi j/N) 6 a_j]
        // (src/cond_opt.cpp:3204-3308)
        if (grp < 2) {
            const double2 d0 = d0s[grp], dN = dNs[grp];
            if (t == 0) {
                const double2 v0 = X[0], vN = X[pidx(N)];
                sC1[grp] = make_double2(-v0.x - vN.x, -v0.y - vN.y);
                sC2[grp] = cadd(d0, dN);
            }
            group_sync<G>(grp);
            spline_complex<N>(X, NJ, t, grp, h, d0, dN, a.spl_full, a.spl_full + NJ);
            if (t == 0) {
                const double2 m0 = X[0], mN = X[pidx(N)];
                sC3[grp] = make_double2(-(m0.x + mN.x), -(m0.y + mN.y));
            }
            auto in = [&](int j) -> double2 {
                const double2 u = X[pidx(j)], v = X[pidx(j + 1)];
                return cmul(tw_at(ht2, j), make_double2((v.x - u.x) * ih, (v.y - u.y) * ih));
            };
            group_fft_io<N, +1, false, true>(X, t, (const TwoLevelTw *)tw2, grp, in, ScratchIO{X});
        }
        __syncthreads();
        // ---- J0(i k_n), J(i k_n), G(i k_n); sum_n G^2 J0; G J and G minus tails
        // in their places; k0, dG/dtau, dJ/dtau sums (src/cond_opt.cpp:3236-3407)
        {
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int n = tid; n < NO; n += NT) {
                const int i0 = pidx(n), i1 = pidx(N - 1 - n);
                // the pre-twiddled split: F_b = (Z_n - conj Z_{N-1-n}) / (2i)
                double2 F0[2], F[2];
                split_real(X1[i0], X1[i1], F0[0], F0[1]);
                split_real(X2[i0], X2[i1], F[0], F[1]);
                const double kn = (2 * n + 1) * pT, ik = 1.0 / kn, ik2 = ik * ik, ik4 = ik2 * ik2;
                const double2 e = tw_at(ht2, 2 * n + 1);
                const double2 f = make_double2(1.0 - e.x, -e.y);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const CondCol &s = col[q];
                    // J(i k_n) = -i C1/k_n - C2/k_n^2 + i C3/k_n^3 + f F/k_n^4, n >= 0
                    const double2 w0 = cmul(f, F0[q]), w = cmul(f, F[q]);
                    const double2 J0 = make_double2(-part_of(sC2[0], q) * ik2 + w0.x * ik4,
                                                    -part_of(sC1[0], q) * ik + part_of(sC3[0], q) * ik2 * ik + w0.y * ik4);
                    const double C1 = part_of(sC1[1], q);
                    const double2 J = make_double2(-part_of(sC2[1], q) * ik2 + w.x * ik4,
                                                   -C1 * ik + part_of(sC3[1], q) * ik2 * ik + w.y * ik4);
                    double rS, iS;
                    sigma_full(ik, sinf, __ldg(&a.s2[s.o]), __ldg(&a.s3[s.o]), a.S[bidx(n, s.o, NO)], rS, iS);
                    const double2 Gv = crecip(T, mu - s.e - rS, kn - iS);
                    const double2 Gt = crecip(T, mu - s.e, kn + sinf * ik);
                    const double2 Gs = csub(Gv, Gt);
                    const double2 Js = csub(cmul(Gv, J), cmul(Gt, make_double2(0.0, -C1 * ik)));
                    acc[4 * q] += cmul(cmul(Gv, Gv), J0).x;
                    acc[4 * q + 1] += Gs.x;
                    acc[4 * q + 2] += kn * Gs.y;
                    acc[4 * q + 3] -= kn * Js.y;
                    X1[q == 0 ? i0 : i1] = Gs;
                    X2[q == 0 ? i0 : i1] = Js;
                }
            }
            block_sum<8>(acc, sums);
        }
        if (tid < 2) {
            const CondCol &c = col[tid];
            ColState &q = cs[tid];
            const double C1 = part_of(sC1[1], tid), *s = sums + 4 * tid;
            q.v1 = cscale(c.w1, C1);
            q.v2 = cscale(c.w2, C1);
            q.q0 = 2.0 * s[0] / T;
            q.k0 = 2.0 * s[1] + c.k0;
            q.dGm = -2.0 * s[2] + c.dGm;
            q.dGp = 2.0 * s[2] + c.dGp;
            q.dJb = -2.0 * s[3] + C1 * c.dJb;
            q.dJ0 = 2.0 * s[3] + C1 * c.dJ0;
        }
        // ---- back to tau: G(tau) = sum_n G(ikn) e^{-ikn tau}, J(tau) = sum_n J(ikn) e^{+ikn tau}
        // (src/cond_opt.cpp:3545-3620); both real, so the pair packs as Re/Im
        if (grp < 2) {
            auto in = [&](int k) -> double2 {
                double2 A, B;
                if (k < NO) {
                    A = X[pidx(k)];
                    B = X[pidx(N - 1 - k)];
                } else {
                    A = cconj(X[pidx(N - 1 - k)]);
                    B = cconj(X[pidx(k)]);
                }
                return make_double2(A.x - B.y, A.y + B.x);
            };
            if (grp == 0)
                group_fft_io<N, -1, false, true>(X, t, (const TwoLevelTw *)tw2, grp, in, ScratchIO{X});
            else
                group_fft_io<N, +1, false, true>(X, t, (const TwoLevelTw *)tw2, grp, in, ScratchIO{X});
        }
        __syncthreads();
        // ---- G(tau) into X1, G J(tau) into X2
        for (int j = tid; j < N; j += NT) {
            const double2 ph = tw_at(ht2, j);
            const double2 g = cmul(cconj(ph), X1[pidx(j)]);
            const double2 jr = cmul(ph, X2[pidx(j)]);
            double g0[2], ji[2];
            if (real_roots) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const CondCol &c = col[q];
                    auto E = [&](int k, int jj) -> double {
                        return tails_hi[(2 * q + k) * P::n_hi + (jj >> 6)] * tails_lo[(2 * q + k) * P::n_lo + (jj & 63)];
                    };
                    // r > 0: e = exp(-r tau), j = exp(-r (beta - tau)); r <= 0: the other way round
                    const double a1 = E(0, j), b1 = E(0, N - j), a2 = E(1, j), b2 = E(1, N - j);
                    const bool big1 = c.r1.x > 0, big2 = c.r2.x > 0;
                    g0[q] = -c.u1.x * (big1 ? a1 : b1) - c.u2.x * (big2 ? a2 : b2);
                    ji[q] = cs[q].v1.x * (big1 ? b1 : a1) + cs[q].v2.x * (big2 ? b2 : a2);
                }
            } else {
                tails(col[0], cs[0], j * h, beta, g0[0], ji[0]);
                tails(col[1], cs[1], j * h, beta, g0[1], ji[1]);
            }
            const double Ga = g.x + g0[0], Gb = g.y + g0[1], Ja = jr.x + ji[0], Jb = jr.y + ji[1];
            X2[pidx(j)] = make_double2(Ga * Ja, Gb * Jb);
            X1[pidx(j)] = make_double2(Ga, Gb);
            if (j == 0) {
                cs[0].Gt0 = Ga;
                cs[1].Gt0 = Gb;
                cs[0].Jt0 = Ja;
                cs[1].Jt0 = Jb;
                cs[0].Jraw0 = jr.x;
                cs[1].Jraw0 = jr.y;
            }
        }
        __syncthreads();
        // ---- the bubble -G(tau) G(beta - tau) on [0, beta/2] in X1 (node j reads
        // nodes j and N - j, and only it does; src/cond_opt.cpp:3662-3700), the
        // end node and slopes of both splines
        {
            KSum va, vb;
            for (int j = tid; j <= NO; j += NT) {
                double2 v;
                if (j == 0) {
                    v = make_double2(cs[0].Gt0 * (cs[0].Gt0 + 1.0), cs[1].Gt0 * (cs[1].Gt0 + 1.0));
                } else {
                    const double2 g = X1[pidx(j)], gm = X1[pidx(N - j)];
                    v = make_double2(-g.x * gm.x, -g.y * gm.y);
                }
                X1[pidx(j)] = v;
                // trapezoid weights
                const double w = (j == 0 || j == NO) ? 0.5 : 1.0;
                va.add(w * v.x);
                vb.add(w * v.y);
            }
            if (tid < 2) {
                ColState &q = cs[tid];
                double g0b, jinfb;
                tails(col[tid], q, beta, beta, g0b, jinfb);
                const double Jbeta = -q.Jraw0 + jinfb;  // J(beta) = -sum_n J(ikn) + Jinf(beta)
                const double vN = (-q.Gt0 - 1.0) * Jbeta;
                q.CJ1b = q.Gt0 * q.Jt0 - vN;
                q.dchi = q.dGp * (q.Gt0 + 1.0) + q.Gt0 * q.dGm;
                double *xN = reinterpret_cast<double *>(&X2[pidx(N)]);
                double *s0 = reinterpret_cast<double *>(d0s), *sN = reinterpret_cast<double *>(dNs);
                xN[tid] = vN;
                s0[tid] = q.dchi;
                sN[tid] = 0.0;
                s0[2 + tid] = q.dGp * q.Jt0 + q.Gt0 * q.dJ0;
                sN[2 + tid] = q.dGm * Jbeta - (q.Gt0 + 1.0) * q.dJb;
            }
            KSum v2[2] = {va, vb};
            block_ksum<2>(v2, sV);
        }
        // ---- splines and FFT_{-} of both: the bubble's moments from the half
        // spline (odd about beta/2), the Maki-Thompson moment from the G J
        // spline (src/cond_opt.cpp:3622-3660, 3784-3817)
        if (grp == 0) {
            spline_complex<N>(X1, NJ2, t, 0, h, d0s[0], dNs[0], a.spl_half, a.spl_half + NJ2);
            KSum ma, mb;
            for (int j = t; j <= NO; j += G) {
                const double2 m = X1[pidx(j)];
                const double w = (j == 0 || j == NO) ? 0.5 : 1.0;
                ma.add(w * m.x);
                mb.add(w * m.y);
            }
            constexpr int W = G < 32 ? G : 32;
            const unsigned lanes = G < 32 ? (1u << G) - 1u : 0xffffffffu;
            ma.join_lanes<W>(lanes);
            mb.join_lanes<W>(lanes);
            __shared__ double2 red[2][(G + 31) / 32];
            if (t % 32 == 0) {
                red[0][t / 32] = make_double2(ma.s, ma.c);
                red[1][t / 32] = make_double2(mb.s, mb.c);
            }
            auto in = [&](int j) -> double2 {
                const bool lo = j < NO;
                const int jj = lo ? j : N - 1 - j;
                const double sg = lo ? ih : -ih;
                const double2 u = X1[pidx(jj)], v = X1[pidx(jj + 1)];
                return make_double2((v.x - u.x) * sg, (v.y - u.y) * sg);
            };
            group_fft_io<N, -1, false, true>(X1, t, (const TwoLevelTw *)tw2, 0, in, ScratchIO{X1});
            if (t < 2) {
                for (int q = t; q < 2; q += G) {
                    KSum sM;
                    for (int w = 0; w < (G + 31) / 32; ++w) sM.join(red[q][w].x, red[q][w].y);
                    cs[q].integ = h * sV[q] - h * h * h / 12.0 * sM.value();
                }
            }
        } else if (grp == 1) {
            spline_complex<N>(X2, NJ, t, 1, h, d0s[1], dNs[1], a.spl_full, a.spl_full + NJ);
            if (t == 0) {
                const double2 m0 = X2[0], mN = X2[pidx(N)];
                cs[0].CJ3b = m0.x - mN.x;
                cs[1].CJ3b = m0.y - mN.y;
            }
            auto in = [&](int j) -> double2 {
                const double2 u = X2[pidx(j)], v = X2[pidx(j + 1)];
                return make_double2((v.x - u.x) * ih, (v.y - u.y) * ih);
            };
            group_fft_io<N, -1, false, true>(X2, t, (const TwoLevelTw *)tw2, 1, in, ScratchIO{X2});
        }
        __syncthreads();
        const bool same = col[0].bin == col[1].bin;
        for (int n = 1 + tid; n <= NO; n += NT) {
            double2 Fb[2], F[2];
            split_real(X1[pidx(n)], X1[pidx(N - n)], Fb[0], Fb[1]);
            split_real(X2[pidx(n)], X2[pidx(N - n)], F[0], F[1]);
            const double wq = 2 * n * pT, iw = 1.0 / wq, iw2 = iw * iw, iw4 = iw2 * iw2;
            const double2 e = tw_at(tw2, n);
            const double2 f = make_double2(1.0 - e.x, -e.y);
            double b[2], m[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const CondCol &c = col[q];
                const ColState &s = cs[q];
                const double imJ = -2.0 * s.CJ1b * iw + 2.0 * s.CJ3b * iw2 * iw + 2.0 * cmul(f, F[q]).y * iw4;
                const double bub = -2.0 * s.dchi * iw2 + cmul(f, Fb[q]).x * iw4;
                m[q] = nf * c.wt * c.dk * imJ * iw;
                b[q] = 2.0 * c.wt * nf * c.dk * c.dk * bub;
            }
            double *p0 = part + col[0].bin * PWB + n;
            if (same) {
                p0[0] -= b[0] + b[1];
                p0[NJ2] -= m[0] + m[1];
            } else {
                double *p1 = part + col[1].bin * PWB + n;
                p0[0] -= b[0];
                p0[NJ2] -= m[0];
                p1[0] -= b[1];
                p1[NJ2] -= m[1];
            }
        }
        if (tid == 0) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const CondCol &c = col[q];
                const ColState &s = cs[q];
                part[c.bin * PWB] -= 2.0 * c.wt * nf * c.dk * c.dk * (2.0 * s.integ);
                part[c.bin * PWB + NJ2] -= nf * c.wt * c.dk * s.q0;
                part[a.pw - 1] -= 2.0 * c.wt * nf * c.d2 * s.k0;
            }
        }
        __syncthreads();
    }
}

// kx0 on the kx = 0 and kx = pi lines (src/cond_opt.cpp:3993-4173): one block
// per (line, m); lines[i] = -2 w nf d2eps/dkx2 [sum_n (G - Gtail) + tail roots]
__global__ void __launch_bounds__(256)
    k_cond_lines(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                 const double *__restrict__ sinfp, const double *__restrict__ ek, const double *__restrict__ d2line,
                 int nbk, int nw0, double mu, double T, double nf, double *__restrict__ lines) {
    const int i = blockIdx.x;
    const int l = i < nbk ? 0 : nbk - 1, m = i % nbk;
    const int o = oct_index(l, m), NO = nw0 / 2;
    const double sinf = sinfp[0], e = ek[o], pT = kPi * T;
    double v[1] = {0.0};
    for (int n = threadIdx.x; n < NO; n += blockDim.x) {
        const double kn = (2 * n + 1) * pT, ik = 1.0 / kn;
        double rS, iS;
        sigma_full(ik, sinf, s2[o], s3[o], S[bidx(n, o, NO)], rS, iS);
        const double2 Gv = cdiv(make_double2(T, 0.0), make_double2(mu - e - rS, kn - iS));
        const double2 Gt = cdiv(make_double2(T, 0.0), make_double2(mu - e, kn + sinf * ik));
        v[0] += Gv.x - Gt.x;
    }
    __shared__ double tot[1];
    block_sum<1>(v, tot);
    if (threadIdx.x == 0) {
        double2 r1, r2;
        roots_2pol(make_double2(mu - e, 0.0), make_double2(-sinf, 0.0), r1, r2);
        const double2 a1 = cdiv(r1, csub(r1, r2)), a2 = cdiv(r2, csub(r2, r1));
        auto fm = [&](double2 r, double2 av) -> double2 {
            if (r.x > 0) {
                const double2 ex = cexp2(cscale(r, -1.0 / T));
                return cdiv(cmul(av, ex), make_double2(ex.x + 1.0, ex.y));
            }
            const double2 ex = cexp2(cscale(r, 1.0 / T));
            return cdiv(av, make_double2(ex.x + 1.0, ex.y));
        };
        const double kk = 2.0 * tot[0] + (fm(r1, a1).x + fm(r2, a2).x);
        const double w = (m == 0 || m == nbk - 1) ? 1.0 : 2.0;
        lines[i] = -2.0 * w * nf * d2line[i] * kk;
    }
}

// Sum the per-CTA rows: out = [binned (nbins x 2 NB)], [totals chijj1 (NB),
// chijj2 (NB)], [kx0].  A block takes 32 columns of a bin row, its warps a
// segment of the rows each (compensated), added in warp order: deterministic.
// Block 0 of x = gridDim.x - 1 takes kx0.  One thread per column walked all rows
// before: 69 us at 256^2 x 4096 with three bins, 19 now.
constexpr int kCondFinishWarps = 16;
__global__ void __launch_bounds__(32 * kCondFinishWarps)
    k_cond_finish(const double *__restrict__ partial, int nblk, int pw, int nbins, int PWB,
                  const double *__restrict__ lines, int nlines, double *__restrict__ out) {
    __shared__ double2 seg[kCondFinishWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x == gridDim.x - 1) {
        KSum s;
        for (int b = threadIdx.x; b < nblk + nlines; b += blockDim.x)
            s.add(b < nblk ? partial[(size_t)b * pw + pw - 1] : lines[b - nblk]);
        KSum v[1] = {s};
        __shared__ double tot[1];
        block_ksum<1>(v, tot);
        if (threadIdx.x == 0) out[(size_t)nbins * PWB + PWB] = tot[0];
        return;
    }
    const int i = blockIdx.x * 32 + lane;
    const int per = (nblk + kCondFinishWarps - 1) / kCondFinishWarps, b0 = warp * per, b1 = min(nblk, b0 + per);
    KSum tot;
    for (int bin = 0; bin < nbins; ++bin) {
        KSum s;
        if (i < PWB)
#pragma unroll 4
            for (int b = b0; b < b1; ++b) s.add(partial[(size_t)b * pw + bin * PWB + i]);
        seg[warp][lane] = make_double2(s.s, s.c);
        __syncthreads();
        if (warp == 0 && i < PWB) {
            KSum a;
            for (int w = 0; w < kCondFinishWarps; ++w) {
                a.add(seg[w][lane].x);
                a.add(seg[w][lane].y);
            }
            const double v = a.value();
            out[(size_t)bin * PWB + i] = v;
            tot.add(v);
        }
        __syncthreads();
    }
    if (warp == 0 && i < PWB) out[(size_t)nbins * PWB + i] = tot.value();
}

// ---------------------------------------------------------------------------
// batched continued-fraction Pade (Vidberg-Serene), one CTA per function:
// g_0(l) = y_l, g_m(l) = (g_{m-1}(m-1) - g_{m-1}(l)) / ((x_l - x_{m-1}) g_{m-1}(l)),
// a_m = g_m(m) (generique::pade_cont_frac_coef_rec, src/generique.cpp:1649-1663),
// computed in shared memory, one barrier per order m; then every thread
// evaluates the continued fraction at its energies with the recurrence of
// generique::pade (src/generique.cpp:1628-1646).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_pade_batch(const double2 *__restrict__ x, const double2 *__restrict__ y, int Nn, const double2 *__restrict__ z,
                 int Nz, double2 *__restrict__ out) {
    extern __shared__ __align__(16) double2 sp[];
    double2 *xs = sp, *g = sp + Nn;
    const int f = blockIdx.x;
    for (int l = threadIdx.x; l < Nn; l += blockDim.x) {
        xs[l] = x[(size_t)f * Nn + l];
        g[l] = y[(size_t)f * Nn + l];
    }
    __syncthreads();
    for (int m = 1; m < Nn; ++m) {
        const double2 gm = g[m - 1], xm = xs[m - 1];
        for (int l = m + threadIdx.x; l < Nn; l += blockDim.x)
            g[l] = cdiv(csub(gm, g[l]), cmul(csub(xs[l], xm), g[l]));
        __syncthreads();
    }
    for (int iz = threadIdx.x; iz < Nz; iz += blockDim.x) {
        const double2 zz = z[iz];
        double2 A = make_double2(1.0, 0.0);
        double2 B = cadd(make_double2(1.0, 0.0), cmul(csub(zz, xs[0]), g[1]));
        double2 q = cdiv(A, B);
        for (int j = 3; j <= Nn; ++j) {
            const double2 t = cmul(csub(zz, xs[j - 2]), g[j - 1]);
            A = cadd(make_double2(1.0, 0.0), cdiv(t, A));
            B = cadd(make_double2(1.0, 0.0), cdiv(t, B));
            q = cdiv(cmul(q, A), B);
        }
        out[(size_t)f * Nz + iz] = cmul(q, g[0]);
    }
}

// ---------------------------------------------------------------------------
// launch wrappers per compiled size
// ---------------------------------------------------------------------------
template <int NBK>
struct RunCondSlices {
    // ny = 2: the h and f0 slices and all four end conditions; ny = 1: h only
    static cudaError_t run(const GridDev *g, const CondDev *c, const double *V, const double *dchirt0, double mu0,
                           double T, double fact, int ny, bool f32, cudaStream_t st) {
        const size_t sm = SlicePlan<NBK>::bytes, smw = SliceSmem<NBK, SliceGroups<NBK>::wide>::bytes;
        cudaError_t e = set_smem(k_cond_slice<NBK>, sm);
        if (e != cudaSuccess) return e;
        if ((e = set_smem(k_cond_boundary<NBK>, smw)) != cudaSuccess) return e;
        const double nf = 1.0 / ((double)g->nk0 * g->nk0);
        k_cond_table<<<(c->K4 + 255) / 256, 256, 0, st>>>(g->ek, c->dek, c->K4, g->nbk, mu0, T, nf, c->tab);
        if ((e = launched()) != cudaSuccess) return e;
        if (f32) {
            if ((e = launch_cond_slice32(*g, *c, V, T, ny, st)) != cudaSuccess) return e;
        } else {
            k_cond_slice<NBK><<<dim3(g->nw0 + 1, ny), SlicePlan<NBK>::threads, sm, st>>>(c->tab, V, g->tw_k, g->nw0, T,
                                                                                c->K4p, c->hV, c->f0V, c->pre);
            if ((e = launched()) != cudaSuccess) return e;
        }
        k_cond_boundary<NBK><<<2 * ny, kSliceThreads, smw, st>>>(g->ek, c->dek, V, dchirt0, g->tw_k, c->pre, g->nw0, c->K4p,
                                                            mu0, T, nf, fact, c->dbound);
        return launched();
    }
};

template <int N>
struct RunCondTau {
    static cudaError_t run(const GridDev *g, const CondDev *c, const double2 *S, const double *s2, const double *s3,
                           const double *sinf, double mu, double T, cudaStream_t st) {
        const size_t sm = CondTauPlan<N>::bytes;
        cudaError_t e = set_smem(k_cond_tau<N>, sm);
        if (e != cudaSuccess) return e;
        CondCol *cols = reinterpret_cast<CondCol *>(c->cols);
        k_cond_cols<<<(c->K4p + 63) / 64, 64, 0, st>>>(g->ek, c->dek, c->d2ek, c->nbins > 1 ? c->bin : nullptr, sinf,
                                                       c->K4, c->K4p, g->nbk, mu, T, cols);
        if ((e = launched()) != cudaSuccess) return e;
        CondTauArgs a;
        a.hV = reinterpret_cast<const double2 *>(c->hV);
        a.f0V = reinterpret_cast<const double2 *>(c->f0V);
        a.dbound = c->dbound;
        a.S = S;
        a.s2 = s2;
        a.s3 = s3;
        a.sinf = sinf;
        a.cols = cols;
        a.spl_full = g->spl_full;
        a.spl_half = g->spl_half;
        a.tw = g->tw_w;
        a.ht = g->ht_w;
        a.partial = c->partial;
        a.K4 = c->K4;
        a.K4p = c->K4p;
        a.pw = c->pw;
        a.mu = mu;
        a.T = T;
        a.nf = 1.0 / ((double)g->nk0 * g->nk0);
        const size_t pbytes = (size_t)c->nblk * c->pw * sizeof(double);
        if ((e = cudaMemsetAsync(c->partial, 0, pbytes, st)) != cudaSuccess) return e;
        k_cond_tau<N><<<c->nblk, CondTauPlan<N>::threads, sm, st>>>(a);
        return launched();
    }
};

template <int N>
struct CondBlocks {
    static cudaError_t run(int *blocks) {
        cudaError_t e = set_smem(k_cond_tau<N>, CondTauPlan<N>::bytes);
        if (e != cudaSuccess) return e;
        int dev = 0, sms = 0, per = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cond_tau<N>, CondTauPlan<N>::threads,
                                                          CondTauPlan<N>::bytes);
        if (e != cudaSuccess) return e;
        *blocks = sms * (per > 0 ? per : 1);
        return cudaSuccess;
    }
};

}  // namespace

size_t cond_col_words() { return kCondColWords; }

cudaError_t cond_blocks(const GridDev &g, int *blocks) { return dispatch_nw<CondBlocks>(g.nw0, blocks); }

cudaError_t launch_cond_model(const GridDev &g, const CondDev &c, double tp, double tpp, double t3, cudaStream_t st) {
    const int n = c.K4 + 2 * g.nbk;
    k_cond_model<<<(n + 255) / 256, 256, 0, st>>>(g.ktab, g.nbk, c.K4, tp, tpp, t3, c.dek, c.d2ek, c.d2line);
    return launched();
}

cudaError_t launch_cond_table(const GridDev &g, const CondDev &c, double mu0, double T, cudaStream_t st) {
    const double nf = 1.0 / ((double)g.nk0 * g.nk0);
    k_cond_table<<<(c.K4 + 255) / 256, 256, 0, st>>>(g.ek, c.dek, c.K4, g.nbk, mu0, T, nf, c.tab);
    return launched();
}

cudaError_t launch_cond_slices(const GridDev &g, const CondDev &c, const double *V, const double *dtau_chirt0,
                               double mu0, double T, double fact, cudaStream_t st) {
    return dispatch_nbk<RunCondSlices>(g.nbk, &g, &c, V, dtau_chirt0, mu0, T, fact, 2, false, st);
}

cudaError_t launch_cond_slices32(const GridDev &g, const CondDev &c, const double *V, const double *dtau_chirt0,
                                 double mu0, double T, double fact, cudaStream_t st) {
    return dispatch_nbk<RunCondSlices>(g.nbk, &g, &c, V, dtau_chirt0, mu0, T, fact, 2, true, st);
}

cudaError_t launch_cond_slices_h(const GridDev &g, const CondDev &c, const double *V, const double *dtau_chirt0,
                                 double mu0, double T, double fact, cudaStream_t st) {
    return dispatch_nbk<RunCondSlices>(g.nbk, &g, &c, V, dtau_chirt0, mu0, T, fact, 1, false, st);
}

cudaError_t launch_cond_tau(const GridDev &g, const CondDev &c, const double2 *S, const double *s2, const double *s3,
                            const double *sinf, double mu, double T, cudaStream_t st) {
    return dispatch_nw<RunCondTau>(g.nw0, &g, &c, S, s2, s3, sinf, mu, T, st);
}

cudaError_t launch_pade_batch(const double2 *x, const double2 *y, int nf, int Nn, const double2 *z, int Nz,
                              double2 *out, cudaStream_t st) {
    if (nf < 1 || Nn < 2 || Nn > kPadeBatchMax || Nz < 1) return cudaErrorInvalidValue;
    const size_t sm = (size_t)2 * Nn * sizeof(double2);
    cudaError_t e = set_smem(k_pade_batch, sm);
    if (e != cudaSuccess) return e;
    k_pade_batch<<<nf, 256, sm, st>>>(x, y, Nn, z, Nz, out);
    return launched();
}

cudaError_t launch_cond_finish(const GridDev &g, const CondDev &c, const double2 *S, const double *s2,
                               const double *s3, const double *sinf, double mu, double T, cudaStream_t st) {
    const double nf = 1.0 / ((double)g.nk0 * g.nk0);
    k_cond_lines<<<2 * g.nbk, 256, 0, st>>>(S, s2, s3, sinf, g.ek, c.d2line, g.nbk, g.nw0, mu, T, nf, c.lines);
    cudaError_t e = launched();
    if (e != cudaSuccess) return e;
    const int PWB = 2 * (g.nw0 / 2 + 1);
    k_cond_finish<<<(PWB + 31) / 32 + 1, 32 * kCondFinishWarps, 0, st>>>(c.partial, c.nblk, c.pw, c.nbins, PWB, c.lines, 2 * g.nbk,
                                                          c.out);
    return launched();
}

}  // namespace tpsc
