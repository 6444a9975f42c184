// tpsc_roots.cu -- the root searches on the device: the Newton form's, then the
// reference form's (find_zero, tpsc_findzero.h, over the same grid-wide sums) and
// the Fermi-surface hot spot's.
//
// The Newton form's: the sum-rule roots Usp and Uch (chi::find_Usp_Uch(nq0, nw0, Usc),
// src/chi.cpp:846-876) as one cooperative kernel: every block sums its share
// of the stored frequencies below the series cut, a grid barrier, then every
// block adds the partials and the high-frequency moment series and takes the
// same safeguarded Halley step (the pass also sums the second derivative),
// until both roots have converged.  One launch and one readback replace a
// host round trip per evaluation.
//
// The grid barrier spins on a generation counter with a wall-time bound:
// the launch is cooperative (every block resident), so the bound only ends
// a wait for blocks that are off the GPU all that time; it then sets the error
// flag, every block leaves, and the host repeats the search in one block.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tpsc_device.cuh"
#include "tpsc_findzero.h"

namespace tpsc {

namespace {

constexpr int kRootThreads = 256;
constexpr int kRootMaxNb = 2049;  // bosonic frequencies of Nw0 = 4096
// wall time a barrier wait spins before it gives up (%globaltimer, ns)
constexpr unsigned long long kBarrierNs = 1500000000ull;

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// The grid barrier: bar[0] counts arrivals, bar[1] is the generation (read
// once: it grows by one per barrier).  sync() returns false (and sets *err)
// when the wait ran out or another block had already failed.  The arrival is
// one acq_rel atomic and the waiting thread polls the generation with acquire
// loads, without sleeping: the barrier opens within about one L2 round trip of
// the last arrival.  The error word and the clock are looked at only every
// 64th poll.  (With fences around a plain atomic, the generation and the error
// word read at every barrier and the clock at every poll, an evaluation of the
// sum-rule search cost 1.3 us more.)
struct GridBar {
    unsigned *bar;
    int *err;
    unsigned gen;
    __device__ GridBar(unsigned *bar_, int *err_) : bar(bar_), err(err_), gen(*(volatile unsigned *)(bar_ + 1)) {}
    __device__ bool sync() {
        __shared__ int s_ok;
        __syncthreads();
        const int ok = sync_warp0();
        if (threadIdx.x == 0) s_ok = ok;
        __syncthreads();
        return s_ok;
    }
    // by a block's first warp alone, for what its lane 0 has written: the result in lane 0
    __device__ int sync_warp0() {
        int ok = 1;
        ++gen;
        if (threadIdx.x == 0) {
            unsigned old;
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
            if (old == gridDim.x - 1) {
                asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(bar), "r"(0) : "memory");
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar + 1) : "memory");
            } else {
                unsigned long long t0 = 0;
                for (unsigned i = 1;; ++i) {
                    unsigned g;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(g) : "l"(bar + 1) : "memory");
                    if (g == gen) break;
                    if (i % 64) continue;
                    const unsigned long long t = globaltimer_ns();
                    if (!t0) t0 = t;
                    if (*(volatile int *)err || t - t0 > kBarrierNs) {
                        atomicExch(err, 1);
                        ok = 0;
                        break;
                    }
                }
            }
        }
        return ok;
    }
};

// Grid-stride walk over the items it = blk * nj + j (blk a column block,
// j < nj a frequency): both indices are stepped by the stride's quotient and
// remainder, so that no item pays a 64-bit division.  nj <= 0: no items.
struct GridWalk {
    int blk, j, dblk, dj, nj;
    __device__ explicit GridWalk(int nj_) : nj(nj_) {
        if (nj <= 0) {
            blk = 0x7fffffff;
            j = dblk = dj = 0;
            return;
        }
        const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        const long long stride = (long long)gridDim.x * blockDim.x;
        blk = (int)(first / nj);
        j = (int)(first - (long long)blk * nj);
        dblk = (int)(stride / nj);
        dj = (int)(stride - (long long)dblk * nj);
    }
    // the item after (b, jj) in this thread's walk
    __device__ void after(int b, int jj, int &nb, int &nj2) const {
        nb = b + dblk;
        nj2 = jj + dj;
        if (nj2 >= nj) {
            nj2 -= nj;
            ++nb;
        }
    }
};

struct RootCtl {
    double x, lo, hi, prev_step, root;
    int nev, it, done, ok;
};

struct SumRootArgs {
    const double4 *chiq;
    const double *cinf, *cinf2, *w16, *tailq;
    const double *mom_suf;   // [(nb + 1) kMomP] sums of the moments over frequencies >= j
    const double *cmax_suf;  // [nb + 1] max |chi| over frequencies >= j
    const double *tailm;     // [kMomP] tail moments, [kMomP] = max |chi| over the tail
    int nb, nblk, n8;
    double T, scale, n, nsr, U, hi_sp;
    const double *chi0max;  // device max chi0(q, 0), or null: hi_sp as given
    double hi_off;          // hi_sp = 2 / chi0max - hi_off
    double *partial;  // [kRootPartial]: two buffers of kRootVals values per block, or of one per
                      // column block (k_sumrule_zero), or the slots (k_sumrule_slots)
    unsigned *bar;    // [2], zero at launch
    int *err;         // zero at launch
    double *out;      // Usp, Uch, evals_sp, evals_ch, ok_sp, ok_ch
    Bp b;             // batched launch: point blockIdx.z, blocks blockIdx.x of gridDim.x per point
    int cached;       // (k_sumrule_slots) column blocks of a block whose rows are kept in its shared memory
};

// the value and its derivatives, each summed in a fixed order, into
// dst[0..kRootVals)
__device__ void block_root_sums(double v, double dv, double d2v, double *dst) {
    __shared__ double red[32][kRootVals];
    for (int off = 16; off > 0; off >>= 1) {
        v += __shfl_down_sync(0xffffffffu, v, off);
        dv += __shfl_down_sync(0xffffffffu, dv, off);
        d2v += __shfl_down_sync(0xffffffffu, d2v, off);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5][0] = v;
        red[threadIdx.x >> 5][1] = dv;
        red[threadIdx.x >> 5][2] = d2v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0, c = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            a += red[w][0];
            b += red[w][1];
            c += red[w][2];
        }
        dst[0] = a;
        dst[1] = b;
        dst[2] = c;
    }
    __syncthreads();
}

// warp 0 adds every block's partials of one evaluation in the same order
__device__ void grid_root_sums(const double *part, double &pv, double &pd, double &p2) {
    pv = pd = p2 = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) {
        pv += __ldcg(&part[kRootVals * b]);
        pd += __ldcg(&part[kRootVals * b + 1]);
        p2 += __ldcg(&part[kRootVals * b + 2]);
    }
    for (int off = 16; off > 0; off >>= 1) {
        pv += __shfl_down_sync(0xffffffffu, pv, off);
        pd += __shfl_down_sync(0xffffffffu, pd, off);
        p2 += __shfl_down_sync(0xffffffffu, p2, off);
    }
}

// One safeguarded update with the bracket, bisection fallback and stopping
// tests of a safeguarded Newton search ([lo, hi] shrinks to the side that the
// signs of the value and the derivative leave; converged when |f| is below
// tol, when the step is below 1e-14 relative, or when it stops shrinking while
// below 1e-10 relative: f is then at its rounding floor).  The step is
// Halley's, x - 2 y y' / (2 y'^2 - y y''), while |y y''| <= y'^2 (it is then
// between 2/3 and 2 Newton steps); else, and with d2y = 0, Newton's.
__device__ void newton_update(RootCtl &c, double y, double dy, double tol, double d2y = 0.0) {
    ++c.nev;
    if (!isfinite(y) || !isfinite(dy)) {
        c.done = 1;
        c.ok = 0;
        return;
    }
    if (fabs(y) < tol) {
        c.root = c.x;
        c.done = c.ok = 1;
        return;
    }
    if ((y > 0) == (dy > 0))
        c.hi = fmin(c.hi, c.x);
    else
        c.lo = fmax(c.lo, c.x);
    const double scale = fmax(1.0, fabs(c.x));
    double xn = 0.5 * (c.lo + c.hi);
    if (dy != 0.0) {
        const double yy = y * d2y, dd = dy * dy;
        xn = (d2y != 0.0 && fabs(yy) <= dd) ? c.x - 2.0 * y * dy / (2.0 * dd - yy) : c.x - y / dy;
    }
    if (dy != 0.0 && fabs(xn - c.x) <= 1e-14 * scale) {
        c.root = xn;
        c.done = c.ok = 1;
        return;
    }
    if (!(xn >= c.lo && xn <= c.hi)) xn = 0.5 * (c.lo + c.hi);
    const double step = fabs(xn - c.x);
    if (c.it >= 2 && step < 1e-10 * scale && step > 0.5 * c.prev_step) {
        c.root = xn;
        c.done = c.ok = 1;
        return;
    }
    c.prev_step = step;
    c.x = xn;
    if (++c.it >= 60) {
        c.done = 1;
        c.ok = 0;
    }
}

// One barrier per evaluation: every block writes its partial sums into the
// buffer of the iteration's parity, waits at the barrier, then adds ALL
// partials in the same order and takes the same Newton step on its own copy
// of the state (identical in every block).  A buffer is rewritten two
// iterations later, after a barrier that every reader of it has passed.
//
// The spin search iterates on s = -ln(1 - Us/hi), hi = 2/chi0max - 2 eps,
// Us = -hi expm1(-s): R_sp has the AFM pole at hi and behaves like -ln of the
// distance to it, so Newton in Us overshoots the pole and falls back to
// bisection step after step, while in s it converges in a few steps.  The
// root is the same zero of R_sp.
constexpr double kSpinSMax = 40.0;  // -hi expm1(-40) = hi (1 - 4e-18)

__device__ __forceinline__ double spin_us(double s, double hi) { return -hi * expm1(-s); }

__global__ void __launch_bounds__(kRootThreads) k_sumrule_roots(SumRootArgs a) {
    {
        const long long ar = a.b.arena;
        a.chiq = at(a.chiq, ar);
        a.cinf = at(a.cinf, ar);
        a.cinf2 = at(a.cinf2, ar);
        a.tailq = at(a.tailq, ar);
        a.mom_suf = at(a.mom_suf, ar);
        a.cmax_suf = at(a.cmax_suf, ar);
        a.tailm = at(a.tailm, ar);
        a.chi0max = at(a.chi0max, ar);
        a.partial = at(a.partial, ar);
        a.bar = at(a.bar, ar);
        a.err = at(a.err, ar);
        a.out = at(a.out, ar);
        a.T = bpar(a.b, kPpT, a.T);
        a.scale = bpar(a.b, kPpNormFact, a.scale);
        a.n = bpar(a.b, kPpN, a.n);
        a.nsr = bpar(a.b, kPpNsr, a.nsr);
        a.U = bpar(a.b, kPpU, a.U);
    }
    // the spin interval's upper end 2/chi0max - 2 eps, from the device maximum
    // when the chi0 stage left it there (no host round trip)
    const double hi_sp = a.chi0max ? 2.0 / a.chi0max[0] - a.hi_off : a.hi_sp;
    __shared__ RootCtl sc;
    __shared__ int s_jdir, s_tail;
    // cmax_suf and tailm staged once; the series moments of an evaluation's
    // cut are fetched before its pass and read after the barrier
    __shared__ double s_cmax[kRootMaxNb], s_tailm[kMomP + 1], s_M[kMomP];
    for (int j = threadIdx.x; j < a.nb; j += blockDim.x) s_cmax[j] = a.cmax_suf[j];
    for (int m = threadIdx.x; m <= kMomP; m += blockDim.x) s_tailm[m] = a.tailm[m];
    const int nwmax = a.nb - 1;
    const double tw = 2.0 * 3.141592653589793 * a.T;
    double Usp = 0.0;
    int parity = 0;
    GridBar bar(a.bar, a.err);
#pragma unroll 1
    for (int phase = 0; phase < 2; ++phase) {
        const double sgn = phase == 0 ? -1.0 : 1.0;
        if (threadIdx.x == 0) {
            const double hi = phase == 0 ? hi_sp : 1000.0 * a.U;
            // spin: U/2 (clamped inside the interval); charge: U
            const double x0 = phase == 0 ? a.U / 2.0 : a.U;
            const double xs = (x0 > 0.0 && x0 < hi) ? x0 : 0.5 * hi;
            sc.lo = 0.0;
            sc.hi = phase == 0 ? kSpinSMax : hi;
            sc.x = phase == 0 ? -log1p(-xs / hi) : xs;
            sc.prev_step = 0.0;
            sc.nev = sc.it = sc.done = sc.ok = 0;
        }
        __syncthreads();
#pragma unroll 1
        while (!sc.done) {
            if (threadIdx.x < 32) {
                const double ah = fabs(phase == 0 ? spin_us(sc.x, hi_sp) : sc.x) / 2.0;
                // first frequency of the series (cmax_suf does not increase):
                // every j < lo is below the cut and every j >= hi above it;
                // a round probes 32 points of [lo, hi) and keeps one step of it
                int lo = 0, hi = a.nb;
                while (hi > lo) {
                    const int step = (hi - lo + 31) / 32;
                    const int q = lo + ((int)threadIdx.x + 1) * step - 1;
                    const bool below = q < hi && ah * s_cmax[q] >= kMomSeriesMax;
                    const int t = __popc(__ballot_sync(0xffffffffu, below));
                    const int qt = lo + (t + 1) * step - 1;
                    if (t < 32 && qt < hi) hi = qt;
                    lo += t * step;
                }
                const bool tail = ah * s_tailm[kMomP] >= kMomSeriesMax;
                if (threadIdx.x < kMomP)
                    s_M[threadIdx.x] = (lo < a.nb ? a.mom_suf[(size_t)lo * kMomP + threadIdx.x] : 0.0) +
                                       (tail ? 0.0 : s_tailm[threadIdx.x]);
                if (threadIdx.x == 0) {
                    s_jdir = lo;
                    s_tail = tail;
                }
            }
            __syncthreads();
            const double x = phase == 0 ? spin_us(sc.x, hi_sp) : sc.x, hu = sgn * x / 2.0;
            const int jdir = s_jdir;
            // v = sum f w (q - x), q = x / (1 + h x), h = sgn U / 2; its U
            // derivatives: dq/dU = -sgn q^2 / 2, d2q/dU2 = q^3 / 2
            double v = 0.0, dv = 0.0, d2v = 0.0;
            // the next item's chi0 row is loaded before this item's arithmetic
            const GridWalk walk(jdir);
            int blk = walk.blk, j = walk.j;
            double4 xn = blk < a.nblk ? a.chiq[(size_t)blk * a.nb + j] : make_double4(0.0, 0.0, 0.0, 0.0);
            while (blk < a.nblk) {
                const double4 xq = xn;
                int nb, nj;
                walk.after(blk, j, nb, nj);
                if (nb < a.nblk) xn = a.chiq[(size_t)nb * a.nb + nj];
                const double4 w = reinterpret_cast<const double4 *>(a.w16)[blk];
                const double f = j == 0 ? 0.5 : 1.0;
                const double xs[4] = {xq.x, xq.y, xq.z, xq.w}, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double q = xs[c] / (1.0 + hu * xs[c]), fw = f * ws[c];
                    v += fw * (q - xs[c]);
                    dv += fw * q * q;
                    d2v += fw * q * q * q;
                }
                blk = nb;
                j = nj;
            }
            dv *= -0.5 * sgn;
            d2v *= 0.5;
            if (s_tail) {
                // the Matsubara tail term by term (the series does not converge there)
                for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < a.n8; o += gridDim.x * blockDim.x) {
                    const double w = a.w16[o];
                    if (w == 0.0) continue;
                    const double ca = a.cinf[o], cb = a.cinf2[o];
                    for (int t = 0; t < nwmax; ++t) {
                        const double wn = (nwmax + 1 + t) * tw;
                        const double i2 = 1.0 / (wn * wn);
                        const double xv = ca * i2 + cb * i2 * i2;
                        const double q = xv / (1.0 + hu * xv);
                        v += w * (q - xv);
                        dv += w * (-0.5 * sgn) * q * q;
                        d2v += w * 0.5 * q * q * q;
                    }
                }
            }
            double *part = a.partial + (size_t)parity * kRootVals * kRootMaxBlocks;
            block_root_sums(v, dv, d2v, part + kRootVals * blockIdx.x);
            if (!bar.sync()) return;
            parity ^= 1;
            if (threadIdx.x < 32) {
                double pv, pd, p2;
                grid_root_sums(part, pv, pd, p2);
                if (threadIdx.x == 0) {
                    // the series over the frequencies from jdir (and over the
                    // tail), S = sum_m (-h)^m M_m, and its h derivatives
                    double S = 0.0, dS = 0.0, d2S = 0.0, hm1 = 1.0, hm2 = 0.0;  // (-h)^(m-1), (-h)^(m-2)
                    const double h = hu;
                    for (int m = 1; m <= kMomP; ++m) {
                        const double M = s_M[m - 1];
                        S += -h * hm1 * M;
                        dS += -m * hm1 * M;
                        d2S += m * (m - 1) * hm2 * M;
                        hm2 = hm1;
                        hm1 *= -h;
                    }
                    // dh/dU = sgn / 2
                    const double tr = a.scale * (pv + S), dtr = a.scale * (pd + 0.5 * sgn * dS),
                                 d2tr = a.scale * (p2 + 0.25 * d2S);
                    const double n = a.n, nsr = a.nsr, U = a.U;
                    double y, dy, d2y;
                    if (phase == 0) {
                        // chi::sum_rule_sp (src/chi.cpp:833-836)
                        y = tr + n - n * n / 2.0 - nsr + x * nsr * nsr / (2.0 * U);
                        // d/ds = d/dUs * dUs/ds, dUs/ds = hi e^-s = hi - Us,
                        // d2Us/ds2 = -(hi - Us)
                        dy = (dtr + nsr * nsr / (2.0 * U)) * (hi_sp - x);
                        d2y = d2tr * (hi_sp - x) * (hi_sp - x) - dy;
                    } else {
                        // chi::sum_rule_ch (src/chi.cpp:840-843)
                        y = tr + n - n * n / 2.0 - (nsr + Usp * nsr * nsr / (2.0 * U) - nsr * nsr);
                        dy = dtr;
                        d2y = d2tr;
                    }
                    newton_update(sc, y, dy, 1e-16, d2y);
                }
            }
            __syncthreads();
        }
        const double root = phase == 0 ? spin_us(sc.root, hi_sp) : sc.root;
        if (phase == 0) Usp = root;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.out[phase] = root;
            a.out[2 + phase] = sc.nev;
            a.out[4 + phase] = sc.ok;
        }
        if (!sc.ok) return;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// chemical potential
// ---------------------------------------------------------------------------

// One pass over Sigma for the Newton form: Tr Sigma G0 with its asymptotic
// correction (green::traceSelfG, src/green.cpp:3001-3084) over the stored
// frequencies, and the moments of the find_mu series over the stored
// frequencies n >= jc and the tail Nw0/2 <= n <= Nw0 (asymptotic Sigma, as
// green::traceDiffG sums them):
//   C_m = sum w z^-(m+1),  z = i w_n - eps + mu0 - Sigma,  m < kMuMomP,
//   G0  = sum w Re 1/(i w_n - eps + mu0),
// so that this part of Tr(G - G0) at mu is Re sum_m (mu0 - mu)^m C_m - G0 to
// a relative kMuSeriesMax^kMuMomP while |mu - mu0| <= kMuSeriesMax |z|.
//
// C_m for m >= kMuMomF64 is formed and summed in FP32 (per thread: 32 terms of the
// stored frequencies, a column's Nw0/64 + 1 of the tail term by term; the sums of
// columns, blocks and the grid are FP64): its term (mu0 - mu)^m C_m is at most
// kMuSeriesMax^m = 8e-7 of the leading one per point, so an FP32 relative
// error ~1e-6 on it moves Tr(G - G0) by < 1e-12 of its leading term.  The
// point constants live in shared memory and Tr Sigma G0, its Hartree part and
// G0 share one reciprocal per (k, n), so that two CTAs fit on an SM.
//
// Blocks 0 .. take per_s column blocks each over the stored frequencies, their rows
// as one sequence; the four columns of a row are formed without a branch (a padding
// column has weight 0 and finite stand-in values), so that their chains interleave.
// The blocks after them take the tail, half a warp per column and per_t columns one
// after the other, away from the Sigma stream.  Per-block partials (block_store).
// The reduction of a block's kSigmaMomNV sums and, below 256 frequencies, the threads
// without a row were most of a small-cutoff point's time at one column block per block
// and one tail column per warp: at 64 points of a sweep (129 lines, 64 to 1024
// frequencies) 1731 us for its 18 groups, against 960 (256^2 x 4096: 170 -> 149).
constexpr int kMuMomF64 = 4;
constexpr int kTailR = 28;           // terms of the tail power series (needs kMuMomP + kTailR < kTailP)
constexpr double kTailRatio = 0.05;  // series when rho / w_NO < this: terms below 0.05^28 (~1e-36) relative
static_assert(kMuMomP + kTailR < kTailP, "tail power sums too short");
constexpr int kMomThreads = 256;
constexpr int kMomTailCols = kMomThreads / 16;  // columns of a tail block at a time
constexpr int kMomPerMax = 32;                  // column blocks of a block
constexpr int kMomRows = 8;                     // rows of a thread (32 terms, as the FP32 sums allow)

__global__ void __launch_bounds__(kMomThreads, 2)
    k_sigma_moments(const double2 *__restrict__ S, const double *__restrict__ s2, const double *__restrict__ s3,
                    const double *__restrict__ s4, const double *__restrict__ sinfp, const double *__restrict__ ek,
                    const double *__restrict__ w16, const double *__restrict__ tailP, int nw0, double mu0,
                    double T, double nk02, int jc, int nblk, int per_s, int per_t, double *partial, Bp b) {
    constexpr int NV = kSigmaMomNV, P64 = kMuMomF64, P32 = kMuMomP - kMuMomF64;
    __shared__ double cw[4 * kMomPerMax], cx[4 * kMomPerMax], c2[4 * kMomPerMax], c3[4 * kMomPerMax];
    __shared__ __align__(16) double2 s_row[2][kMomThreads][4];  // two stages of 64-byte Sigma rows
    S = at(S, b.arena);
    s2 = at(s2, b.arena);
    s3 = at(s3, b.arena);
    s4 = at(s4, b.arena);
    sinfp = at(sinfp, b.arena);
    ek = at(ek, b.arena);
    tailP = at(tailP, b.arena);
    partial = at(partial, b.arena);
    mu0 = bpar(b, kPpMu0, mu0);
    T = bpar(b, kPpT, T);
    jc = (int)bpar(b, kPpJc, (double)jc);
    const int NO = nw0 / 2, nsb = (nblk + per_s - 1) / per_s;  // blocks of the stored frequencies
    const double sinf = sinfp[0];
    const double pt = 3.141592653589793 * T;
    double tsg = 0.0, har = 0.0, g0 = 0.0;
    double m64[2 * P64];
    float m32[2 * P32];
#pragma unroll
    for (int k = 0; k < 2 * P64; ++k) m64[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 2 * P32; ++k) m32[k] = 0.0f;
    // the FP32 moments of a tail block: their sums, and those of its columns term by term
    // (a thread's at t32[k][threadIdx.x], in place of the Sigma rows: in registers they
    // spilled)
    double a32[2 * P32];
    bool slow_any = false;
    double(*const t32)[kMomThreads] = reinterpret_cast<double(*)[kMomThreads]>(s_row);
    static_assert(sizeof(s_row) >= 2 * P32 * kMomThreads * sizeof(double), "the tail's sums do not fit");
    // z = i w_n - x - Sigma with x = eps - mu0; inv = 1 / (w_n^2 + x^2)
    // rr = 1/|z|^2 (|z| >= w_n > 0)
    auto moments_rr = [&](double zx, double zy, double rr, double x, double w, double inv) {
        const double2 zi = make_double2(zx * rr, -zy * rr);
        double2 zp = zi;
#pragma unroll
        for (int m = 0; m < P64; ++m) {
            m64[2 * m] += w * zp.x;
            m64[2 * m + 1] += w * zp.y;
            zp = cmul(zp, zi);
        }
        const float wf = (float)w;
        const float2 zf = make_float2((float)zi.x, (float)zi.y);
        float2 zq = make_float2((float)zp.x, (float)zp.y);
#pragma unroll
        for (int m = 0; m < P32; ++m) {
            m32[2 * m] += wf * zq.x;
            m32[2 * m + 1] += wf * zq.y;
            zq = make_float2(zq.x * zf.x - zq.y * zf.y, zq.x * zf.y + zq.y * zf.x);
        }
        g0 -= w * x * inv;
    };
    auto moments = [&](double wn, double rS, double iS, double x, double w, double inv) {
        const double zx = -x - rS, zy = wn - iS;
        moments_rr(zx, zy, 1.0 / (zx * zx + zy * zy), x, w, inv);
    };
    double fermi = 0.0;  // traceSelfG's Fermi-function term of a stored-frequency block's columns
    if ((int)blockIdx.x < nsb) {
        const int blk0 = blockIdx.x * per_s, o0 = 4 * blk0, ncb = min(per_s, nblk - blk0), ncol = 4 * ncb;
        if ((int)threadIdx.x < ncol) {
            // a padding column: weight 0, x = 1 and Sigma's coefficients 0,
            // so that |z| and w_n^2 + x^2 stay away from 0 and its terms are 0
            const int c = threadIdx.x;
            const double w = w16[o0 + c];
            const bool ok = w != 0.0;
            cw[c] = w;
            cx[c] = ok ? ek[o0 + c] - mu0 : 1.0;
            c2[c] = ok ? s2[o0 + c] : 0.0;
            c3[c] = ok ? s3[o0 + c] : 0.0;
        }
        __syncthreads();
        // this thread's Sigma rows tid + 256 i of the block's column blocks through
        // two shared-memory stages: row i + 1 is copied (cp.async, 4 x 16 bytes)
        // while row i is formed; each thread reads back only its own copies
        const double2 *row = S + (size_t)blk0 * 4 * NO;
        const int nrow = ncb * NO, lno = 31 - __clz(NO);  // NO is a power of two
        auto issue = [&](int jj, int st) {
#pragma unroll
            for (int c = 0; c < 4; ++c) cp_async16(&s_row[st][threadIdx.x][c], row + 4 * (size_t)jj + c);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        if ((int)threadIdx.x < nrow) issue(threadIdx.x, 0);
        for (int i = threadIdx.x, st = 0; i < nrow; i += blockDim.x, st ^= 1) {
            const int j = i & (NO - 1), cb = 4 * (i >> lno);
            const double wn = (2 * j + 1) * pt, i1 = 1.0 / wn;
            if (i + (int)blockDim.x < nrow) {
                issue(i + blockDim.x, st ^ 1);
                asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            }
            const double2 sv[4] = {s_row[st][threadIdx.x][0], s_row[st][threadIdx.x][1], s_row[st][threadIdx.x][2],
                                   s_row[st][threadIdx.x][3]};
            if (j >= jc) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double w = cw[cb + c], x = cx[cb + c];
                    const double2 s = w != 0.0 ? sv[c] : make_double2(0.0, 0.0);
                    double rS, iS;
                    sigma_full(i1, sinf, c2[cb + c], c3[cb + c], s, rS, iS);
                    // one reciprocal for 1/(w_n^2 + x^2) and 1/|z|^2
                    const double b = wn * wn + x * x;
                    const double zx = -x - rS, zy = wn - iS, a = zx * zx + zy * zy;
                    const double r = 1.0 / (a * b), inv = r * a;
                    tsg += w * inv * (rS * (-x) + iS * wn);
                    har += w * inv;
                    moments_rr(zx, zy, r * b, x, w, inv);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double w = cw[cb + c], x = cx[cb + c];
                    const double2 s = w != 0.0 ? sv[c] : make_double2(0.0, 0.0);
                    double rS, iS;
                    sigma_full(i1, sinf, c2[cb + c], c3[cb + c], s, rS, iS);
                    const double inv = 1.0 / (wn * wn + x * x);
                    tsg += w * inv * (rS * (-x) + iS * wn);
                    har += w * inv;
                }
            }
        }
        // traceSelfG's Fermi-function term per octant point
        if ((int)threadIdx.x < ncol) {
            const int c = threadIdx.x;
            const double w8 = 0.5 * cw[c];
            if (w8 != 0.0) {
                const double x = cx[c];
                if (fabs(x) > 1.0e-12) {
                    fermi = w8 * sinf * (1.0 / (exp(x / T) + 1.0) - 0.5) / x / nk02;
                } else {
                    const double ex = (x < 0) ? exp(x / T) : exp(-x / T);
                    fermi = -w8 * sinf * ex / ((ex + 1.0) * (ex + 1.0) * nk02 * T);
                }
            }
        }
    } else {
        // The tail n = NO .. 2 NO (asymptotic Sigma), half a warp for column o:
        // with u = 1/(i w_n), z^-1 = u / (1 - q(u)), q(u) = x u + Sinf u^2 +
        // C2 u^3 + C3 u^4 + C4 u^5 (real coefficients), and h^(p) the
        // coefficients of (1 - q)^-p,
        //   sum_tail z^-p = sum_r h^(p)_r (-i)^(p+r) P_(p+r),
        //   sum_tail Re 1/(i w_n - x) = -x sum_k (-x^2)^k P_(2k+2),
        // P_p = sum_tail w_n^-p (tailP).  (1 - q)^-p obeys H' (1 - q) = p q' H,
        // so R h_R = sum_{s=1..5} q_s h_(R-s) (R - s + p s),   h_0 = 1:
        // lane p - 1 of the half runs the recurrence of moment m = p - 1 in registers
        // and keeps the sum over its columns.  The terms fall like (rho / w_NO)^r, rho
        // a bound on q's root radius; above kTailRatio the warp sums term by term.
        static_assert(kMuMomP < 16, "the moments and G0 of a column in half a warp");
        const int lane = threadIdx.x & 31, sub = lane & 15, half = threadIdx.x >> 4;
        const double w_no = (2 * NO + 1) * pt;
        double sre = 0.0, sim = 0.0;  // lanes sub < kMuMomP: w C_sub, sub = kMuMomP: w G0
        for (int r = 0; r < per_t; ++r) {
            const int o = ((blockIdx.x - nsb) * per_t + r) * kMomTailCols + half;
            const double w = o < 4 * nblk ? __ldg(&w16[o]) : 0.0;
            double x = 0.0, q3 = 0.0, q4 = 0.0, q5 = 0.0;
            const double q2 = sinf;
            bool series = true;
            if (w != 0.0) {
                x = __ldg(&ek[o]) - mu0;
                q3 = __ldg(&s2[o]);
                q4 = __ldg(&s3[o]);
                q5 = __ldg(&s4[o]);
                const double rho =
                    fabs(x) + sqrt(fabs(sinf)) + cbrt(fabs(q3)) + sqrt(sqrt(fabs(q4))) + pow(fabs(q5), 0.2);
                series = rho < kTailRatio * w_no;
                if (series) {
                    double re = 0.0, im = 0.0;
                    if (sub < kMuMomP) {
                        const double p = sub + 1;
                        // h_(R-1) .. h_(R-5) in a register window
                        double h1 = 1.0, h2 = 0.0, h3 = 0.0, h4 = 0.0, h5 = 0.0;
                        // r = 0 term: (-i)^p P_p
                        auto add = [&](int k, double h) {
                            const double t = h * __ldg(&tailP[k]);
                            switch (k & 3) {
                                case 0: re += t; break;
                                case 1: im -= t; break;
                                case 2: re -= t; break;
                                default: im += t; break;
                            }
                        };
                        add(sub + 1, 1.0);
                        // unrolled: 1 / R is a constant of each step
#pragma unroll
                        for (int R = 1; R <= kTailR; ++R) {
                            const double hR = (x * h1 * (R - 1 + p) + q2 * h2 * (R - 2 + 2 * p) +
                                               q3 * h3 * (R - 3 + 3 * p) + q4 * h4 * (R - 4 + 4 * p) +
                                               q5 * h5 * (R - 5 + 5 * p)) *
                                              (1.0 / R);
                            add(sub + 1 + R, hR);
                            h5 = h4;
                            h4 = h3;
                            h3 = h2;
                            h2 = h1;
                            h1 = hR;
                        }
                    } else if (sub == kMuMomP) {
                        // G0: -x sum_k (-x^2)^k P_(2k+2)
                        double xp = 1.0;
                        for (int k = 0; 2 * k + 2 < kTailP; ++k, xp *= -x * x) re += xp * __ldg(&tailP[2 * k + 2]);
                        re *= -x;
                    }
                    sre += w * re;
                    sim += w * im;
                }
            }
            // the columns of the warp that the series does not hold for
            const unsigned slow = __ballot_sync(0xffffffffu, !series);
            for (int hf = 0; hf < 2; ++hf)
                if (slow >> (16 * hf) & 1u) {
                    const double wc = __shfl_sync(0xffffffffu, w, 16 * hf), xc = __shfl_sync(0xffffffffu, x, 16 * hf);
                    const double a3 = __shfl_sync(0xffffffffu, q3, 16 * hf), a4 = __shfl_sync(0xffffffffu, q4, 16 * hf),
                                 a5 = __shfl_sync(0xffffffffu, q5, 16 * hf);
                    for (int t = lane; t <= NO; t += 32) {
                        const double wn = (2 * (NO + t) + 1) * pt, i1 = 1.0 / wn, i2 = i1 * i1;
                        moments(wn, -a3 * i2 + a5 * i2 * i2, -sinf * i1 + a4 * i2 * i1, xc, wc,
                                1.0 / (wn * wn + xc * xc));
                    }
#pragma unroll
                    for (int k = 0; k < 2 * P32; ++k) {
                        t32[k][threadIdx.x] = m32[k] + (slow_any ? t32[k][threadIdx.x] : 0.0);
                        m32[k] = 0.0f;
                    }
                    slow_any = true;
                }
        }
        sre += __shfl_down_sync(0xffffffffu, sre, 16);
        sim += __shfl_down_sync(0xffffffffu, sim, 16);
#pragma unroll
        for (int m = 0; m < kMuMomP; ++m) {
            const double rm = __shfl_sync(0xffffffffu, sre, m), imm = __shfl_sync(0xffffffffu, sim, m);
            if (m < P64) {
                m64[2 * m] += lane == 0 ? rm : 0.0;
                m64[2 * m + 1] += lane == 0 ? imm : 0.0;
            } else {
                a32[2 * (m - P64)] = lane == 0 ? rm : 0.0;
                a32[2 * (m - P64) + 1] = lane == 0 ? imm : 0.0;
            }
        }
        if (slow_any)
#pragma unroll
            for (int k = 0; k < 2 * P32; ++k) a32[k] += t32[k][threadIdx.x];
        const double gt = __shfl_sync(0xffffffffu, sre, kMuMomP);
        if (lane == 0) g0 += gt;
    }
    if ((int)blockIdx.x < nsb)
#pragma unroll
        for (int k = 0; k < 2 * P32; ++k) a32[k] = m32[k];
    double acc[NV];
    acc[0] = tsg * T / nk02;
    acc[1] = har * sinf * T / nk02 + fermi;
#pragma unroll
    for (int k = 0; k < 2 * P64; ++k) acc[2 + k] = m64[k];
#pragma unroll
    for (int k = 0; k < 2 * P32; ++k) acc[2 + 2 * P64 + k] = a32[k];
    acc[2 + 2 * kMuMomP] = g0;
    block_store<NV>(acc, partial);
}

struct MuRootArgs {
    const double2 *S;
    const double *s2, *s3, *s4, *sinf, *ek, *w16;
    const double *mom;  // the k_sigma_moments results
    int nw0, nblk, jc;
    double mu0, T, nk02, wc;  // wc = w_jc
    double *partial;  // as above
    unsigned *bar;
    int *err;
    double *out;  // mu, evals, ok, Tr Sigma G at mu
    Bp b;         // batched launch: point blockIdx.z
    int cached;   // (k_mu_slots) as above, Sigma
};

// the four octant points of column block blk at frequency j of
// green::traceSelfG2 (src/green.cpp:2929-2976): sum w8 2T/nk02 Re[Sigma G]
// with G = 1/(i w_n - e + mu - Sigma); p, q the block's Sigma row at j.  The
// four fractions K N / A share one division: sum K_c N_c / A_c =
// [(K0 N0 A1 + K1 N1 A0) A2 A3 + (K2 N2 A3 + K3 N3 A2) A0 A1] / (A0 A1 A2 A3),
// A_c lies between w_n^2 and ~w_max^2, so the products stay far inside FP64's range.
__device__ __forceinline__ double trsg_row(const MuRootArgs &a, int blk, int j, double4 p, double4 q, double mu,
                                           double sinf, double pt) {
    const int o0 = 4 * blk;
    const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                           make_double2(q.z, q.w)};
    const double wn = (2 * j + 1) * pt, i1 = 1.0 / wn, kT = 2.0 * a.T / a.nk02;
    double K[4], N[4], A[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double w8 = 0.5 * __ldg(&a.w16[o0 + c]);
        // a padding column: weight 0, and e - mu = 1 with Sigma's
        // coefficients 0, so that its A >= 1 and its term is 0
        double e = 1.0, c2 = 0.0, c3 = 0.0;
        double2 s = make_double2(0.0, 0.0);
        if (w8 != 0.0) {
            e = __ldg(&a.ek[o0 + c]) - mu;
            c2 = __ldg(&a.s2[o0 + c]);
            c3 = __ldg(&a.s3[o0 + c]);
            s = sv[c];
        }
        double rS, iS;
        sigma_full(i1, sinf, c2, c3, s, rS, iS);
        const double aa = e + rS;
        A[c] = (wn - iS) * (wn - iS) + aa * aa;
        N[c] = iS * wn - iS * iS - e * rS - rS * rS;
        K[c] = w8 * kT;
    }
    const double P01 = A[0] * A[1], P23 = A[2] * A[3];
    return ((K[0] * N[0] * A[1] + K[1] * N[1] * A[0]) * P23 + (K[2] * N[2] * A[3] + K[3] * N[3] * A[2]) * P01) /
           (P01 * P23);
}

// find_mu by safeguarded Halley steps (newton_update) from
// mu0 inside [-10, 10] with tolerance 1e-15, one barrier per evaluation as in
// k_sumrule_roots; then green::traceSelfG2 (src/green.cpp:2929-2976) at mu.
__global__ void __launch_bounds__(kRootThreads) k_mu_roots(MuRootArgs a) {
    {
        const long long ar = a.b.arena;
        a.S = at(a.S, ar);
        a.s2 = at(a.s2, ar);
        a.s3 = at(a.s3, ar);
        a.s4 = at(a.s4, ar);
        a.sinf = at(a.sinf, ar);
        a.ek = at(a.ek, ar);
        a.mom = at(a.mom, ar);
        a.partial = at(a.partial, ar);
        a.bar = at(a.bar, ar);
        a.err = at(a.err, ar);
        a.out = at(a.out, ar);
        a.mu0 = bpar(a.b, kPpMu0, a.mu0);
        a.T = bpar(a.b, kPpT, a.T);
        a.jc = (int)bpar(a.b, kPpJc, (double)a.jc);
        a.wc = bpar(a.b, kPpWc, a.wc);
    }
    __shared__ RootCtl sc;
    const int NO = a.nw0 / 2;
    const double sinf = a.sinf[0];
    const double pt = 3.141592653589793 * a.T;
    // the series holds while |mu - mu0| <= kMuSeriesMax |z|_min, |z|_min = w_jc - 2 |Sigma_inf| / w_jc
    const double zmin = a.wc - 2.0 * fabs(sinf) / a.wc;
    const double dmax = zmin > 0.0 ? kMuSeriesMax * zmin : 0.0;
    int parity = 0;
    GridBar bar(a.bar, a.err);
    if (threadIdx.x == 0) {
        sc.lo = -10.0;
        sc.hi = 10.0;
        sc.x = (a.mu0 > sc.lo && a.mu0 < sc.hi) ? a.mu0 : 0.0;
        sc.prev_step = 0.0;
        sc.nev = sc.it = sc.done = sc.ok = 0;
    }
    __syncthreads();
#pragma unroll 1
    while (!sc.done) {
        const double pmu = sc.x, delta = pmu - a.mu0;
        const bool series = fabs(delta) <= dmax;
        const int jhi = series ? a.jc : NO;
        double v = 0.0, dv = 0.0, d2v = 0.0;
        const GridWalk walk(jhi);
        for (int blk = walk.blk, j = walk.j; blk < a.nblk; walk.after(blk, j, blk, j)) {
            const int o0 = 4 * blk;
            const double4 *row = reinterpret_cast<const double4 *>(a.S + (size_t)blk * 4 * NO);
            const double4 p = ld_stream4(&row[2 * j]), q = ld_stream4(&row[2 * j + 1]);
            const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                                   make_double2(q.z, q.w)};
            const double wn = (2 * j + 1) * pt, i1 = 1.0 / wn;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double w = __ldg(&a.w16[o0 + c]);
                if (w == 0.0) continue;
                double rS, iS;
                sigma_full(i1, sinf, __ldg(&a.s2[o0 + c]), __ldg(&a.s3[o0 + c]), sv[c], rS, iS);
                trdiff_term(wn, rS, iS, __ldg(&a.ek[o0 + c]), a.mu0, pmu, w, v, dv, d2v);
            }
        }
        if (!series) {
            // the tail Nw0/2 <= n <= Nw0 with the asymptotic Sigma, term by term
            const long long ttot = (long long)a.nblk * 4 * (NO + 1);
            for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < ttot;
                 it += (long long)gridDim.x * blockDim.x) {
                const int o = (int)(it / (NO + 1)), t = (int)(it - (long long)o * (NO + 1));
                const double w = __ldg(&a.w16[o]);
                if (w == 0.0) continue;
                const double wn = (2 * (NO + t) + 1) * pt, i1 = 1.0 / wn, i2 = i1 * i1;
                const double rS = -__ldg(&a.s2[o]) * i2 + __ldg(&a.s4[o]) * i2 * i2;
                const double iS = -sinf * i1 + __ldg(&a.s3[o]) * i2 * i1;
                trdiff_term(wn, rS, iS, __ldg(&a.ek[o]), a.mu0, pmu, w, v, dv, d2v);
            }
        }
        double *part = a.partial + (size_t)parity * kRootVals * kRootMaxBlocks;
        block_root_sums(v, dv, d2v, part + kRootVals * blockIdx.x);
        if (!bar.sync()) return;
        parity ^= 1;
        if (threadIdx.x < 32) {
            double pv, pd, p2;
            grid_root_sums(part, pv, pd, p2);
            if (threadIdx.x == 0) {
                if (series) {
                    // Re sum_m (-delta)^m C_m - G0 and its first two mu derivatives
                    double sr = 0.0, dsr = 0.0, d2sr = 0.0, pr = 1.0, pm = 0.0, pmm = 0.0;
                    for (int m = 0; m < kMuMomP; ++m) {  // pr, pm, pmm = (-delta)^(m, m-1, m-2)
                        const double C = a.mom[2 + 2 * m];
                        sr += pr * C;
                        dsr += -m * pm * C;
                        d2sr += m * (m - 1) * pmm * C;
                        pmm = pm;
                        pm = pr;
                        pr *= -delta;
                    }
                    pv += sr - a.mom[2 + 2 * kMuMomP];
                    pd += dsr;
                    p2 += d2sr;
                }
                newton_update(sc, pv, pd, 1e-15, p2);
            }
        }
        __syncthreads();
    }
    if (!sc.ok) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.out[0] = sc.x;
            a.out[1] = sc.nev;
            a.out[2] = 0.0;
            a.out[3] = 0.0;
        }
        return;
    }
    // Tr Sigma G at mu over the stored frequencies; the next item's Sigma
    // row is loaded before this item's arithmetic.
    const double mu = sc.root;
    double v = 0.0;
    {
        const GridWalk walk(NO);
        int blk = walk.blk, j = walk.j;
        auto load = [&](int bk, int jj, double4 &p, double4 &q) {
            const double4 *row = reinterpret_cast<const double4 *>(a.S + (size_t)bk * 4 * NO);
            p = ld_stream4(&row[2 * jj]);
            q = ld_stream4(&row[2 * jj + 1]);
        };
        double4 p = make_double4(0.0, 0.0, 0.0, 0.0), q = p;
        if (blk < a.nblk) load(blk, j, p, q);
        while (blk < a.nblk) {
            int nb, nj;
            walk.after(blk, j, nb, nj);
            double4 pn = p, qn = q;
            if (nb < a.nblk) load(nb, nj, pn, qn);
            v += trsg_row(a, blk, j, p, q, mu, sinf, pt);
            blk = nb;
            j = nj;
            p = pn;
            q = qn;
        }
    }
    double *part = a.partial + (size_t)parity * kRootVals * kRootMaxBlocks;
    block_root_sums(v, 0.0, 0.0, part + kRootVals * blockIdx.x);
    if (!bar.sync()) return;
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        double pv, pd, p2;
        grid_root_sums(part, pv, pd, p2);
        if (threadIdx.x == 0) {
            a.out[0] = mu;
            a.out[1] = sc.nev;
            a.out[2] = 1.0;
            a.out[3] = pv;
        }
    }
}

// ---------------------------------------------------------------------------
// the reference form's root searches (find_zero, tpsc_findzero.h) on the
// device: every block runs the search on the same function values, one grid
// barrier per evaluation.  The function is the reference's: every stored
// frequency and the Matsubara tail, no series over the stored frequencies.
//
// What bounded the host-driven search is the round trip of an evaluation (the
// sum, its gather into mapped memory, the wait: ~20 us, of which the sum
// itself is 6-8 us up to 64^2 x 1024), 40-60 evaluations a solve; here an
// evaluation costs the pass and one barrier.  The sums are taken in the order
// of k_sumrule and k_trace_diff_G -- one partial per column block, added in
// block order -- so the search sees the same values to the last bit whatever
// the grid (differences of two roots, as the grid-halving diagnostics form
// them, keep their digits).
// ---------------------------------------------------------------------------

// sum over the column blocks of share(blk) over each block's threads, the
// same in every thread of the grid; part: one value per column block.
// False: the barrier ran out.
template <class F>
__device__ bool grid_total(int nblk, double *part, GridBar &bar, double &total, const F &share) {
    __shared__ double red[kRootThreads / 32], s_total;
    for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        double v = share(blk);
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double x = 0.0;
            for (int w = 0; w < kRootThreads / 32; ++w) x += red[w];
            part[blk] = x;
        }
        __syncthreads();
    }
    if (gridDim.x > 1 && !bar.sync()) return false;
    if (threadIdx.x < 32) {
        KSum acc;
        for (int b = threadIdx.x; b < nblk; b += 32) acc.add(__ldcg(&part[b]));
        double x = acc.value();
        for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if (threadIdx.x == 0) s_total = x;
    }
    __syncthreads();
    total = s_total;
    __syncthreads();
    return true;
}

// the tail's power sums of a block's first kZeroTail column blocks, which do
// not depend on U: formed once per search
constexpr int kZeroTail = 16;
struct ZeroTail {
    double S[kZeroTail][4][kTailM];
};

// (not inlined: find_zero evaluates at many places)
__device__ __noinline__ bool sumrule_total(const SumRootArgs &a, const ZeroTail &zt, double Uv, double sgn, double *part,
                                           GridBar &bar, double &tr) {
    const double hu = sgn * Uv / 2.0;
    return grid_total(a.nblk, part, bar, tr, [&](int blk) {
        const double4 w = reinterpret_cast<const double4 *>(a.w16)[blk];
        const double ww[4] = {w.x, w.y, w.z, w.w};
        const int lb = (blk - (int)blockIdx.x) / (int)gridDim.x;
        double v, dv, tv, tdv;
        sumrule_stored<false>(a.chiq, ww, blk, a.nb, a.nb, hu, v, dv);
        sumrule_tail(a.cinf, a.cinf2, ww, blk, a.nb, hu, sgn, a.T, tv, tdv,
                     [&](int c, double ca, double cb, double &f, double &df) {
                         if (lb >= kZeroTail) {
                             tail_series(ca, cb, hu, a.tailq, f, df);
                             return;
                         }
                         f = df = 0.0;
                         double hm = 1.0;
                         for (int m = 1; m <= kTailM; ++m) {
                             f += (-hu) * hm * zt.S[lb][c][m - 1];
                             hm *= -hu;
                         }
                     });
        return a.scale * (v + tv);
    });
}

// Usp and Uch (chi::find_Usp_Uch(nq0, nw0, Usc), src/chi.cpp:850-876) -> out
// as k_sumrule_roots leaves them
__global__ void __launch_bounds__(kRootThreads, 2) k_sumrule_zero(SumRootArgs a) {
    const double hi_sp = a.chi0max ? 2.0 / a.chi0max[0] - a.hi_off : a.hi_sp;
    const double n = a.n, nsr = a.nsr, U = a.U;
    __shared__ ZeroTail zt;
    for (int i = threadIdx.x; i < 4 * kZeroTail; i += blockDim.x) {
        const int o = 4 * (blockIdx.x + (i >> 2) * gridDim.x) + (i & 3);
        if (o < a.n8) tail_sums(a.cinf[o], a.cinf2[o], a.tailq, zt.S[i >> 2][i & 3]);
    }
    __syncthreads();
    GridBar bar(a.bar, a.err);
    int parity = 0;
    double Usp = 0.0;
#pragma unroll 1
    for (int phase = 0; phase < 2; ++phase) {
        const double sgn = phase == 0 ? -1.0 : 1.0;
        auto f = [&](double Uv, double &y) -> bool {
            double tr;
            double *part = a.partial + (size_t)parity * kRootVals * kRootMaxBlocks;
            parity ^= 1;
            if (!sumrule_total(a, zt, Uv, sgn, part, bar, tr)) return false;
            // chi::sum_rule_sp (src/chi.cpp:833-836) and sum_rule_ch (840-843),
            // rounded as the host's expressions
            const Rn base = Rn(tr) + Rn(n) - Rn(n) * Rn(n) / Rn(2.0);
            if (phase == 0)
                y = (base - Rn(nsr) + Rn(Uv) * Rn(nsr) * Rn(nsr) / (Rn(2.0) * Rn(U))).v;
            else
                y = (base - (Rn(nsr) + Rn(Usp) * Rn(nsr) * Rn(nsr) / (Rn(2.0) * Rn(U)) - Rn(nsr) * Rn(nsr))).v;
            return true;
        };
        const double init[3] = {phase == 0 ? U / 2.0 : 0.0, 0.0, phase == 0 ? hi_sp : 1000.0 * U};
        double root = 0.0;
        int nev;
        bool gone;
        const bool ok = find_zero(f, init, &root, nullptr, &nev, &gone);
        if (gone) return;
        if (phase == 0) Usp = root;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.out[phase] = root;
            a.out[2 + phase] = nev;
            a.out[4 + phase] = ok;
        }
        if (!ok) return;
    }
}

__device__ __noinline__ bool trace_diff_total(const MuRootArgs &a, double pmu, double *part, GridBar &bar, double &tr) {
    return grid_total(a.nblk, part, bar, tr, [&](int blk) {
        double v, dv;
        trace_diff_block<false>(a.S, a.s2, a.s3, a.s4, a.sinf, a.ek, a.w16, blk, a.nw0, a.mu0, pmu, a.T, a.nw0 / 2, 1,
                                v, dv);
        return v;
    });
}

// find_mu (src/green.cpp:3185-3259), then traceSelfG2 (src/green.cpp:2929-2976)
// at mu -> out as k_mu_roots leaves them
__global__ void __launch_bounds__(kRootThreads, 2) k_mu_zero(MuRootArgs a) {
    GridBar bar(a.bar, a.err);
    int parity = 0;
    auto buffer = [&]() {
        parity ^= 1;
        return a.partial + (size_t)parity * kRootVals * kRootMaxBlocks;
    };
    auto f = [&](double pmu, double &y) -> bool { return trace_diff_total(a, pmu, buffer(), bar, y); };
    const double init[3] = {0.0, -10.0, 10.0}, lims[2] = {-20.0, 20.0};
    double mu = 0.0;
    int nev;
    bool gone;
    const bool ok = find_zero(f, init, &mu, lims, &nev, &gone);
    if (gone) return;
    double tr = 0.0;
    if (ok && !grid_total(a.nblk, buffer(), bar, tr, [&](int blk) {
            return trace_self2_block<false>(a.S, a.s2, a.s3, a.sinf, a.ek, a.w16, blk, a.nw0, mu, a.T, a.nk02);
        }))
        return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = mu;
        a.out[1] = nev;
        a.out[2] = ok;
        a.out[3] = tr;
    }
}

// Up to kSlotBlocks column blocks: a column block's value goes to every block
// through a slot that a warp of every block polls: one store and one load, where a
// barrier and then a read take an atomic, a store and two loads, behind fences.  A slot
// is two 64-bit words, each half of the value and the number of the evaluation: a word
// is stored and loaded whole, so that no order between words or slots matters and the
// accesses are relaxed (with an empty-slot value instead of the number the stores had to
// release and the loads to acquire, and every kernel's L1 was emptied: 5% slower).
// Two sets of slots in turn: a block stores evaluation e + 2 after it has read all of
// e + 1, which every block stored after it had read e.  kSlotCopies copies of a set, each for as many readers, as one
// would be polled by every SM at once.  With more column blocks every block would
// poll (and wait for) hundreds of slots: there the kernels above are faster
// (537 column blocks: 348 and 324 us a search, with slots 373 and 355).  The lattices
// have 4, 12, 39, 141, 537 and 2097 column blocks: any bound from 141 to 536 is this rule.
constexpr int kSlotBlocks = 148, kSlotCopies = 8, kSlotStride = 160;
static_assert(2 * 2 * kSlotCopies * kSlotStride <= kRootPartial && kSlotStride >= kSlotBlocks, "slots do not fit");
__device__ __forceinline__ void slot_store(ulonglong2 *p, double x, unsigned n) {
    const unsigned long long b = __double_as_longlong(x), t = (unsigned long long)n << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | (b >> 32)), "l"(t | (b & 0xffffffffu))
                 : "memory");
}
// true when the slot holds evaluation n: x
__device__ __forceinline__ bool slot_load(const ulonglong2 *p, unsigned n, double &x) {
    unsigned long long h, l;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(h), "=l"(l) : "l"(p) : "memory");
    x = __longlong_as_double((long long)(h << 32 | (l & 0xffffffffu)));
    return (unsigned)(h >> 32) == n && (unsigned)(l >> 32) == n;
}
struct ZeroSlots {
    ulonglong2 *base;  // [2][kSlotCopies][kSlotStride]
    int nblk;
    unsigned n;  // the evaluation, from 1
    // (the first warp) all slots of evaluation 0, seen by every block
    __device__ bool begin(double *base_, int nblk_, GridBar &bar) {
        base = reinterpret_cast<ulonglong2 *>(base_);
        nblk = nblk_;
        n = 1;
        if (threadIdx.x == 0)
            for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x)
                for (int k = 0; k < 2 * kSlotCopies; ++k) slot_store(base + k * kSlotStride + blk, 0.0, 0);
        return __shfl_sync(0xffffffffu, bar.sync_warp0(), 0);
    }
    __device__ ulonglong2 *slot(int copy, int blk) const {
        return base + ((n & 1) * kSlotCopies + copy) * kSlotStride + blk;
    }
};

// What the first warp asks of a block's threads: an evaluation of kind op at x, or the
// end of the search.  Only that warp runs find_zero; with the search in every thread
// its spilled state, 400 bytes a thread, moved at every evaluation.  The searches for
// Usp and Uch and for mu: 180 and 118 us through barriers at 16^2 x 128, now 119 and
// 78; at 32^2 x 512 224 and 138, now 147 and 61; at 64^2 x 1024 262 and 172, now 210
// and 161 (an evaluation is then 3500 cycles of values, 5700 until the last of 141
// blocks is read, 1400 of find_zero).
struct ZeroCmd {
    double x;
    int op;
};
constexpr int kZeroDone = -1;

// a block's share of the sum: share(blk) over its threads, in thread order, for each of
// its column blocks -> the slots (the first warp)
template <class F>
__device__ __forceinline__ void block_values(int nblk, const ZeroSlots *zs, const F &share) {
    __shared__ double red[kRootThreads / 32];
    for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        double v = share(blk);
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x < kSlotCopies) {
            double x = 0.0;
            for (int w = 0; w < kRootThreads / 32; ++w) x += red[w];
            slot_store(zs->slot(threadIdx.x, blk), x, zs->n);
        }
        if (blk + (int)gridDim.x < nblk) __syncthreads();
    }
}

// (the first warp, after block_values) the sum over the column blocks in block order,
// the same in every block of the grid.  False: a wait ran out (bounded as the barrier's).
__device__ __noinline__ bool slot_total(ZeroSlots &zs, GridBar &bar, double &total) {
    const int nblk = zs.nblk, lane = threadIdx.x & 31;
    const ulonglong2 *mine = zs.slot(blockIdx.x % kSlotCopies, 0);
    constexpr int U = (kSlotBlocks + 31) / 32;
    KSum acc;
    bool ok = true, have[U];
    double v[U];
    unsigned long long t0 = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) have[u] = lane + 32 * u >= nblk || slot_load(mine + lane + 32 * u, zs.n, v[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (lane + 32 * u >= nblk) continue;
        for (unsigned i = 1; ok && !have[u]; ++i) {
            have[u] = slot_load(mine + lane + 32 * u, zs.n, v[u]);
            if (i % 64) continue;
            const unsigned long long t = globaltimer_ns();
            if (!t0) t0 = t;
            if (*(volatile int *)bar.err || t - t0 > kBarrierNs) {
                atomicExch(bar.err, 1);
                ok = false;
            }
        }
        acc.add(v[u]);
    }
    ok = __all_sync(0xffffffffu, ok);
    ++zs.n;
    double x = acc.value();
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    total = __shfl_sync(0xffffffffu, x, 0);
    return ok;
}

// What a block keeps of its column blocks through a search: the chi0 rows (dynamic
// shared memory, of the first a.cached) and, of its first kZeroTail column
// blocks, the weights and the tail's power sums, which do not depend on U, with the
// bound that decides for the series.  The polls' acquire loads empty L1, so that rows
// read from there cost an L2 trip per evaluation.
struct SlotTail {
    double S[kZeroTail][4][kTailM], w[kZeroTail][4], cmax[kZeroTail][4];
};

__device__ __noinline__ void sumrule_values(const SumRootArgs &a, const SlotTail &zt, const double4 *rows, double Uv,
                                            double sgn, const ZeroSlots *zs) {
    const double hu = sgn * Uv / 2.0;
    block_values(a.nblk, zs, [&](int blk) {
        const int lb = (blk - (int)blockIdx.x) / (int)gridDim.x;
        double ww[4];
        bool kept = lb < kZeroTail;
        if (kept) {
#pragma unroll
            for (int c = 0; c < 4; ++c) ww[c] = zt.w[lb][c];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (ww[c] != 0.0 && !(fabs(hu) * zt.cmax[lb][c] < kTailSeriesMax)) kept = false;
        } else {
            const double4 w = reinterpret_cast<const double4 *>(a.w16)[blk];
            ww[0] = w.x;
            ww[1] = w.y;
            ww[2] = w.z;
            ww[3] = w.w;
        }
        double v, dv, tv, tdv;
        const double4 *col = lb < a.cached ? rows + (size_t)lb * a.nb : a.chiq + (size_t)blk * a.nb;
        sumrule_stored<false>(col, ww, 0, a.nb, a.nb, hu, v, dv);
        auto series = [&](int c, double ca, double cb, double &f, double &df) {
            if (lb >= kZeroTail) {
                tail_series(ca, cb, hu, a.tailq, f, df);
                return;
            }
            f = df = 0.0;
            double hm = 1.0;
            for (int m = 1; m <= kTailM; ++m) {
                f += (-hu) * hm * zt.S[lb][c][m - 1];
                hm *= -hu;
            }
        };
        if (kept) {
            // every column by its series, thread c column c
            tv = 0.0;
            if (threadIdx.x < 4 && zt.w[lb][threadIdx.x] != 0.0) {
                double f, df;
                series(threadIdx.x, 0.0, 0.0, f, df);
                tv += zt.w[lb][threadIdx.x] * f;
            }
        } else {
            sumrule_tail(a.cinf, a.cinf2, ww, blk, a.nb, hu, sgn, a.T, tv, tdv, series);
        }
        return a.scale * (v + tv);
    });
}

// Usp and Uch as k_sumrule_zero, through slots
__global__ void __launch_bounds__(kRootThreads, 2) k_sumrule_slots(SumRootArgs a) {
    const double hi_sp = a.chi0max ? 2.0 / a.chi0max[0] - a.hi_off : a.hi_sp;
    const double n = a.n, nsr = a.nsr, U = a.U;
    __shared__ SlotTail zt;
    extern __shared__ __align__(16) double4 zrows[];
    const double tw = 2.0 * 3.141592653589793 * a.T, wn1 = a.nb * tw, x1 = 1.0 / (wn1 * wn1);
    for (int i = threadIdx.x; i < 4 * kZeroTail; i += blockDim.x) {
        const int o = 4 * (blockIdx.x + (i >> 2) * gridDim.x) + (i & 3);
        if (o >= 4 * a.nblk) continue;
        const double w = a.w16[o];
        zt.w[i >> 2][i & 3] = w;
        if (o >= a.n8) continue;
        const double ca = a.cinf[o], cb = a.cinf2[o];
        zt.cmax[i >> 2][i & 3] = fabs(ca) * x1 + fabs(cb) * x1 * x1;
        tail_sums(ca, cb, a.tailq, zt.S[i >> 2][i & 3]);
    }
    for (int blk = blockIdx.x, lb = 0; blk < a.nblk && lb < a.cached; blk += gridDim.x, ++lb)
        for (int j = threadIdx.x; j < a.nb; j += blockDim.x)
            zrows[(size_t)lb * a.nb + j] = a.chiq[(size_t)blk * a.nb + j];
    __syncthreads();
    __shared__ ZeroCmd cmd;
    if (threadIdx.x >= 32) {
        for (;;) {
            __syncthreads();
            if (cmd.op == kZeroDone) return;
            sumrule_values(a, zt, zrows, cmd.x, cmd.op == 0 ? -1.0 : 1.0, nullptr);
        }
    }
    auto ask = [&](int op, double x) {
        if (threadIdx.x == 0) {
            cmd.op = op;
            cmd.x = x;
        }
        __syncthreads();
    };
    GridBar bar(a.bar, a.err);
    ZeroSlots zs;
    bool ok = zs.begin(a.partial, a.nblk, bar);
    double Usp = 0.0;
#pragma unroll 1
    for (int phase = 0; ok && phase < 2; ++phase) {
        auto f = [&](double Uv, double &y) -> bool {
            double tr;
            ask(phase, Uv);
            sumrule_values(a, zt, zrows, Uv, phase == 0 ? -1.0 : 1.0, &zs);
            if (!slot_total(zs, bar, tr)) return false;
            // chi::sum_rule_sp (src/chi.cpp:833-836) and sum_rule_ch (840-843),
            // rounded as the host's expressions
            const Rn base = Rn(tr) + Rn(n) - Rn(n) * Rn(n) / Rn(2.0);
            if (phase == 0)
                y = (base - Rn(nsr) + Rn(Uv) * Rn(nsr) * Rn(nsr) / (Rn(2.0) * Rn(U))).v;
            else
                y = (base - (Rn(nsr) + Rn(Usp) * Rn(nsr) * Rn(nsr) / (Rn(2.0) * Rn(U)) - Rn(nsr) * Rn(nsr))).v;
            return true;
        };
        const double init[3] = {phase == 0 ? U / 2.0 : 0.0, 0.0, phase == 0 ? hi_sp : 1000.0 * U};
        double root = 0.0;
        int nev;
        bool gone;
        ok = find_zero(f, init, &root, nullptr, &nev, &gone);
        if (phase == 0) Usp = root;
        if (!gone && blockIdx.x == 0 && threadIdx.x == 0) {
            a.out[phase] = root;
            a.out[2 + phase] = nev;
            a.out[4 + phase] = ok;
        }
        ok = ok && !gone;
    }
    ask(kZeroDone, 0.0);
}

// zrow: Sigma of the block's column blocks at every frequency of the trace, [lb][4][nw0 + 1]
// (stored ones and the asymptotic tail), of those kept in shared memory
__device__ __noinline__ void trace_diff_values(const MuRootArgs &a, const double2 *zrow, double pmu,
                                               const ZeroSlots *zs) {
    block_values(a.nblk, zs, [&](int blk) {
        double v = 0.0, dv = 0.0;
        const int lb = (blk - (int)blockIdx.x) / (int)gridDim.x;
        if (lb >= a.cached) {
            trace_diff_block<false>(a.S, a.s2, a.s3, a.s4, a.sinf, a.ek, a.w16, blk, a.nw0, a.mu0, pmu, a.T, a.nw0 / 2,
                                    1, v, dv);
            return v;
        }
        // trace_diff_block's terms in its order
        const int NO = a.nw0 / 2, R = a.nw0 + 1;
        const double2 *z = zrow + (size_t)lb * 4 * R;
        const double pt = 3.141592653589793 * a.T;
        double ww[4], e[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            ww[c] = a.w16[4 * blk + c];
            e[c] = ww[c] != 0.0 ? a.ek[4 * blk + c] : 0.0;
        }
        auto row = [&](int j) {
            const double wn = __dmul_rn(2 * j + 1, pt);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (ww[c] == 0.0) continue;
                const double2 q = z[c * R + j];
                trdiff_term(wn, q.x, q.y, e[c], a.mu0, pmu, ww[c], v, dv);
            }
        };
        for (int j = threadIdx.x; j < NO; j += blockDim.x) row(j);
        for (int t = threadIdx.x; t <= NO; t += blockDim.x) row(NO + t);
        return v;
    });
}

// mu and Tr Sigma G as k_mu_zero, through slots
__global__ void __launch_bounds__(kRootThreads, 2) k_mu_slots(MuRootArgs a) {
    extern __shared__ __align__(16) double2 zself[];
    if (a.cached) {
        const int NO = a.nw0 / 2, R = a.nw0 + 1;
        const double sinf = a.sinf[0], pt = 3.141592653589793 * a.T;
        for (int blk = blockIdx.x, lb = 0; blk < a.nblk && lb < a.cached; blk += gridDim.x, ++lb)
            for (int i = threadIdx.x; i < 4 * R; i += blockDim.x) {
                const int j = i >> 2, c = i & 3, o = 4 * blk + c;
                double rS = 0.0, iS = 0.0;
                if (a.w16[o] != 0.0) {
                    const double i1 = 1.0 / __dmul_rn(2 * j + 1, pt);
                    if (j < NO)
                        trdiff_sigma(i1, sinf, a.s2[o], a.s3[o], a.S[((size_t)blk * NO + j) * 4 + c], rS, iS);
                    else
                        trdiff_sigma_tail(i1, sinf, a.s2[o], a.s3[o], a.s4[o], rS, iS);
                }
                zself[((size_t)lb * 4 + c) * R + j] = make_double2(rS, iS);
            }
        __syncthreads();
    }
    __shared__ ZeroCmd cmd;
    auto values = [&](int op, double x, const ZeroSlots *zs) {
        if (op == 0) {
            trace_diff_values(a, zself, x, zs);
            return;
        }
        block_values(a.nblk, zs, [&](int blk) {
            return trace_self2_block<false>(a.S, a.s2, a.s3, a.sinf, a.ek, a.w16, blk, a.nw0, x, a.T, a.nk02);
        });
    };
    if (threadIdx.x >= 32) {
        for (;;) {
            __syncthreads();
            if (cmd.op == kZeroDone) return;
            values(cmd.op, cmd.x, nullptr);
        }
    }
    auto ask = [&](int op, double x) {
        if (threadIdx.x == 0) {
            cmd.op = op;
            cmd.x = x;
        }
        __syncthreads();
    };
    GridBar bar(a.bar, a.err);
    ZeroSlots zs;
    bool ok = zs.begin(a.partial, a.nblk, bar), gone = !ok;
    auto f = [&](double pmu, double &y) -> bool {
        ask(0, pmu);
        trace_diff_values(a, zself, pmu, &zs);
        return slot_total(zs, bar, y);
    };
    const double init[3] = {0.0, -10.0, 10.0}, lims[2] = {-20.0, 20.0};
    double mu = 0.0, tr = 0.0;
    int nev = 0;
    if (ok) ok = find_zero(f, init, &mu, lims, &nev, &gone);
    if (ok && !gone) {
        ask(1, mu);
        values(1, mu, &zs);
        gone = !slot_total(zs, bar, tr);
    }
    if (!gone && blockIdx.x == 0 && threadIdx.x == 0) {
        a.out[0] = mu;
        a.out[1] = nev;
        a.out[2] = ok;
        a.out[3] = tr;
    }
    ask(kZeroDone, 0.0);
}

// mu0 of the finite lattice (green0::find_mu, src/green0.cpp:182-203, 240-262)
// in one block -> result[0], result[1] = 1 when the search succeeded
// The sum is taken in chunks of kMu0Chunk points, each over kMu0Chunk threads (a
// shuffle tree per warp, then a tree over the warps), then over the chunks.
constexpr int kMu0Threads = 1024, kMu0Chunk = 256;
constexpr int kMu0MaxChunks = 64;
__device__ __noinline__ double density_total(const double *__restrict__ ek, int n8, int nbk, double mu, double T,
                                             double nk2, double *wsum, double *tot) {
    const int nchunk = (n8 + kMu0Chunk - 1) / kMu0Chunk, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int WPC = kMu0Chunk / 32;  // warps of a chunk
    for (int o = threadIdx.x; o < nchunk * kMu0Chunk; o += blockDim.x) {
        double v = 0.0;
        if (o < n8) {
            int l, m;
            oct_lm(o, l, m);
            v = 2 * oct_weight(8, l, m, nbk) / ((exp((ek[o] - mu) / T) + 1.0) * nk2);
        }
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) wsum[o >> 5] = v;
    }
    __syncthreads();
    if (warp == 0) {
        double t = 0.0;
        for (int c0 = 0; c0 < nchunk; c0 += 32) {
            double x = 0.0;
            if (c0 + lane < nchunk) {
                const double *w = wsum + (c0 + lane) * WPC;
                x = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
            }
            for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
            t += x;
        }
        if (lane == 0) *tot = t;
    }
    __syncthreads();
    return *tot;
}
__global__ void __launch_bounds__(kMu0Threads)
    k_mu0_zero(const double *__restrict__ ek, int n8, int nbk, double n, double T, double nk2, double *result) {
    static_assert(kMu0Chunk == 256, "density_total's tree over a chunk's eight warps");
    __shared__ double wsum[kMu0MaxChunks * kMu0Chunk / 32], tot;
    auto f = [&](double mu, double &y) -> bool {
        y = density_total(ek, n8, nbk, mu, T, nk2, wsum, &tot) - n;
        return true;
    };
    const double init[3] = {0.0, -8.0, 8.0};
    double root = 0.0;
    int nev;
    bool gone;
    const bool ok = find_zero(f, init, &root, nullptr, &nev, &gone);
    if (threadIdx.x == 0) {
        result[0] = root;
        result[1] = ok;
    }
}

// ---------------------------------------------------------------------------
// the non-interacting Fermi surface's hot spot (green0::find_FS(nk),
// src/green0.cpp:626-676; chi::vF_hot_spots, src/chi.cpp:420-447)
// ---------------------------------------------------------------------------
// eps_k of hamiltonien::dispk (src/hamiltonien.cpp:428-431), rounded as the host rounds it
__device__ double dispk_dev(double kx, double ky, double tp, double tpp, double t3) {
    const Rn cx(cos(kx)), cy(cos(ky));
    Rn e = Rn(-2.0) * (cx + cy) - Rn(4.0) * Rn(tp) * cx * cy;
    if (tpp != 0.0 || t3 != 0.0) {
        const Rn c2x(cos(2 * kx)), c2y(cos(2 * ky));
        e = e - Rn(2.0) * Rn(tpp) * (c2x + c2y) - Rn(4.0) * Rn(t3) * (c2x * cy + c2y * cx);
    }
    return e.v;
}
// On line j, kx - ky = kx0 = j pi/(nk - 1): the root kx in [kx0, pi] of
// eps(kx, kx - kx0) - mu by the bounded find_zero from {(kx0 + pi)/2, kx0, pi} ->
// kx[j], or NaN where there is none.  10001 lines of ~10 evaluations, bound by a host
// thread's latency, took 5 to 10 ms; one thread each, 15 us, and the pair's search
// below 9 us (a scan of 15 temperatures on a 64 x 64 grid: 17.5 -> 4.1 ms).
__global__ void __launch_bounds__(128) k_fermi_lines(int nk, double mu, double tp, double tpp, double t3,
                                                     double *__restrict__ kx) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nk) return;
    const double kx0 = j * kPi / (nk - 1);
    const double init[3] = {0.5 * (kx0 + kPi), kx0, kPi}, lims[2] = {kx0, kPi};
    auto f = [&](double k, double &y) -> bool {
        y = dispk_dev(k, k - kx0, tp, tpp, t3) - mu;
        return true;
    };
    double root = 0.0;
    int nev;
    bool gone;
    const bool ok = find_zero(f, init, &root, lims, &nev, &gone);
    kx[j] = ok ? root : nan("");
}
// The first pair of consecutive points across kx + ky = pi (or the last pair) ->
// out = (kx, ky) of both; from the first line without a root on every point is
// (-1, -1).  One block.
__global__ void __launch_bounds__(1024) k_hot_pair(const double *__restrict__ kx, int nk, double *__restrict__ out) {
    __shared__ int s_end, s_hit;
    if (threadIdx.x == 0) {
        s_end = nk;
        s_hit = nk - 1;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < nk; j += blockDim.x)
        if (isnan(kx[j])) atomicMin(&s_end, j);
    __syncthreads();
    const int end = s_end;
    auto point = [&](int j, double &x, double &y) {
        x = j < end ? kx[j] : -1.0;
        y = j < end ? x - j * kPi / (nk - 1) : -1.0;
    };
    for (int j = threadIdx.x + 1; j < nk - 1; j += blockDim.x) {
        double x1, y1, x2, y2;
        point(j - 1, x1, y1);
        point(j, x2, y2);
        if (!((x1 + y1 - kPi) * (x2 + y2 - kPi) > 0)) atomicMin(&s_hit, j);
    }
    __syncthreads();
    if (threadIdx.x < 2) point(s_hit - 1 + threadIdx.x, out[2 * threadIdx.x], out[2 * threadIdx.x + 1]);
}

// The barrier's bound, exercised: block `withhold` never arrives (negative:
// every block does), so every other block's wait runs out after
// kBarrierNs and leaves with the error flag set.  words[0..1] the barrier,
// words[2] the error flag, words[3] the number of blocks that left with it;
// all zero at launch.
__global__ void __launch_bounds__(kRootThreads) k_barrier_probe(unsigned *words, int withhold) {
    if ((int)blockIdx.x == withhold) return;
    GridBar bar(words, reinterpret_cast<int *>(words + 2));
    const bool ok = bar.sync();
    if (threadIdx.x == 0 && !ok) atomicAdd(words + 3, 1u);
}

// the cooperative grid of the root searches: up to two blocks per SM, or
// `cap` blocks when the caller runs several root searches at once (solver
// streams of a batch), so that all of them fit on the GPU together
template <typename K>
cudaError_t root_grid(K kernel, int *grid, int cap) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kRootThreads, 0)) != cudaSuccess) return e;
    *grid = std::min(sms * std::max(1, std::min(per, 2)), kRootMaxBlocks);
    if (cap > 0) *grid = std::min(*grid, cap);
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_sigma_moments(const GridDev &g, const double2 *S, const double *s2, const double *s3,
                                 const double *s4, const double *sinf, double mu0, double T, int jc, Reduce r,
                                 cudaStream_t st, const Bp &b) {
    // as many column blocks (8 rows a thread at most) and tail columns per block as
    // leave four blocks per SM: fewer reductions and, at small cutoffs, full blocks;
    // at 129 lines and more than 1024 frequencies, or one point of 65 lines and
    // less, one each, as a grid without its last blocks would be slower
    const int nblk = g.n8p / 4, fill = std::max(1, 4 * sm_count());
    auto per = [&](int units, int most) {
        int k = 1;
        while (2 * k <= most && (long long)units * b.P >= 2LL * k * fill) k *= 2;
        return k;
    };
    const int ncols = (4 * nblk + kMomTailCols - 1) / kMomTailCols;  // tail columns, in blocks of kMomTailCols
    const int per_s = per(nblk, std::min(kMomPerMax, std::max(1, kMomRows * kMomThreads / (g.nw0 / 2))));
    const int per_t = per(ncols, 8);
    const int nb = (nblk + per_s - 1) / per_s + (ncols + per_t - 1) / per_t;
    if (nb > kMaxBlocks) return cudaErrorInvalidValue;
    const double nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    k_sigma_moments<<<dim3(nb, 1, b.P), kMomThreads, 0, st>>>(S, s2, s3, s4, sinf, g.ek, g.w16, g.tailP, g.nw0, mu0,
                                                               T, nk02, jc, nblk, per_s, per_t, r.partial, b);
    cudaError_t e = launched();
    if (e != cudaSuccess) return e;
    return finish<kSigmaMomNV>(r, nb, 0.0, st, b);
}

// One block per column block, or per as few of them as the resident grid (or the
// caller's cap) allows: no more blocks than that many rounds need.  *slots: the grid
// exchanges values through slots (few enough column blocks); *cached: those of a
// block's column blocks, col_bytes each, that it then keeps in shared memory with two
// blocks on an SM (100 KB each): all, or none (its loop over both is the slower one).
constexpr size_t kZeroCache = 100 * 1024;
template <typename K>
static cudaError_t zero_grid(K kernel, K with_slots, int nblk, size_t col_bytes, int *grid, int cap, bool *slots,
                             int *cached) {
    *slots = nblk <= kSlotBlocks;
    cudaError_t e = root_grid(*slots ? with_slots : kernel, grid, cap);
    if (e != cudaSuccess) return e;
    const int rounds = (nblk + *grid - 1) / *grid;
    *grid = (nblk + rounds - 1) / rounds;
    *cached = *slots && rounds * col_bytes <= kZeroCache ? rounds : 0;
    if (2LL * nblk > kRootPartial) return cudaErrorInvalidValue;
    return *slots ? set_smem(with_slots, *cached * col_bytes) : cudaSuccess;
}

cudaError_t launch_hot_pair(int nk, double mu, double tp, double tpp, double t3, double *scratch, double *out,
                            cudaStream_t st) {
    k_fermi_lines<<<(nk + 127) / 128, 128, 0, st>>>(nk, mu, tp, tpp, t3, scratch);
    cudaError_t e = launched();
    if (e != cudaSuccess) return e;
    k_hot_pair<<<1, 1024, 0, st>>>(scratch, nk, out);
    return launched();
}

cudaError_t launch_mu0_zero(const GridDev &g, double n, double T, Reduce r, cudaStream_t st) {
    // (few points: few warps, whose barriers are shorter)
    const int chunks = (g.n8 + kMu0Chunk - 1) / kMu0Chunk, threads = std::min(kMu0Threads, chunks * kMu0Chunk);
    if (chunks > kMu0MaxChunks) return cudaErrorInvalidValue;
    k_mu0_zero<<<1, threads, 0, st>>>(g.ek, g.n8, g.nbk, n, T, 4.0 * (g.nbk - 1) * (g.nbk - 1), r.result);
    return launched();
}

cudaError_t launch_mu_zero(const GridDev &g, const double2 *S, const double *s2, const double *s3, const double *s4,
                           const double *sinf, double mu0, double T, RootScratch rs, cudaStream_t st) {
    const int nblk = g.n8p / 4;
    int grid = 0;
    int cached = 0;
    bool slots = false;
    const size_t col_bytes = (size_t)4 * (g.nw0 + 1) * sizeof(double2);
    cudaError_t e = zero_grid(k_mu_zero, k_mu_slots, nblk, col_bytes, &grid, rs.max_blocks, &slots, &cached);
    if (e != cudaSuccess) return e;
    if (rs.reset_mu && (e = cudaMemsetAsync(rs.bar + 4, 0, 2 * sizeof(unsigned) + sizeof(int), st)) != cudaSuccess)
        return e;
    MuRootArgs a{};
    a.S = S;
    a.s2 = s2;
    a.s3 = s3;
    a.s4 = s4;
    a.sinf = sinf;
    a.ek = g.ek;
    a.w16 = g.w16;
    a.nw0 = g.nw0;
    a.nblk = nblk;
    a.mu0 = mu0;
    a.T = T;
    a.nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    a.partial = rs.partial;
    a.bar = rs.bar + 4;
    a.err = reinterpret_cast<int *>(rs.bar + 6);
    a.out = rs.out;
    void *args[] = {&a};
    a.cached = cached;
    e = cudaLaunchCooperativeKernel(slots ? (const void *)k_mu_slots : (const void *)k_mu_zero, dim3(grid), dim3(kRootThreads), args, cached * col_bytes, st);
    if (e != cudaSuccess) return e;
    return launched();
}

cudaError_t launch_sumrule_zero(const GridDev &g, const double *chiq, const double *chi0_inf, const double *chi0_inf2,
                                double T, double n, double nsr, double U, double hi_sp, RootScratch rs,
                                cudaStream_t st, const double *chi0max, double hi_off) {
    const int nblk = g.n8p / 4;
    int grid = 0;
    int cached = 0;
    bool slots = false;
    const size_t col_bytes = (size_t)g.nb * sizeof(double4);
    cudaError_t e = zero_grid(k_sumrule_zero, k_sumrule_slots, nblk, col_bytes, &grid, rs.max_blocks, &slots, &cached);
    if (e != cudaSuccess) return e;
    if (rs.reset_sr && (e = cudaMemsetAsync(rs.bar, 0, 2 * sizeof(unsigned) + sizeof(int), st)) != cudaSuccess)
        return e;
    SumRootArgs a{};
    a.chiq = reinterpret_cast<const double4 *>(chiq);
    a.cinf = chi0_inf;
    a.cinf2 = chi0_inf2;
    a.w16 = g.w16;
    a.tailq = g.tailq;
    a.nb = g.nb;
    a.nblk = nblk;
    a.n8 = g.n8;
    a.T = T;
    a.scale = T / (4.0 * (g.nbk - 1) * (g.nbk - 1));
    a.n = n;
    a.nsr = nsr;
    a.U = U;
    a.hi_sp = hi_sp;
    a.chi0max = chi0max;
    a.hi_off = hi_off;
    a.partial = rs.partial;
    a.bar = rs.bar;
    a.err = reinterpret_cast<int *>(rs.bar + 2);
    a.out = rs.out;
    void *args[] = {&a};
    a.cached = cached;
    e = cudaLaunchCooperativeKernel(slots ? (const void *)k_sumrule_slots : (const void *)k_sumrule_zero, dim3(grid), dim3(kRootThreads), args, cached * col_bytes, st);
    if (e != cudaSuccess) return e;
    return launched();
}

cudaError_t launch_mu_roots(const GridDev &g, const double2 *S, const double *s2, const double *s3, const double *s4,
                            const double *sinf, const double *mom, double mu0, double T, int jc, double wc,
                            RootScratch rs, cudaStream_t st, const Bp &b) {
    int grid = 0;
    cudaError_t e = root_grid(k_mu_roots, &grid, rs.max_blocks);
    if (e != cudaSuccess) return e;
    // a batched search: the resident grid shared out between the points
    // (the caller keeps P at most the resident grid)
    if (b.P > 1) grid = std::max(1, grid / b.P);
    // words 4..6 of rs.bar: the sum-rule search's error flag (word 2) stays readable
    if (rs.reset_mu) {
        e = b.P > 1 ? cudaMemset2DAsync(rs.bar + 4, (size_t)b.arena, 0, 2 * sizeof(unsigned) + sizeof(int), b.P, st)
                    : cudaMemsetAsync(rs.bar + 4, 0, 2 * sizeof(unsigned) + sizeof(int), st);
        if (e != cudaSuccess) return e;
    }
    MuRootArgs a;
    a.S = S;
    a.s2 = s2;
    a.s3 = s3;
    a.s4 = s4;
    a.sinf = sinf;
    a.ek = g.ek;
    a.w16 = g.w16;
    a.mom = mom;
    a.nw0 = g.nw0;
    a.nblk = g.n8p / 4;
    a.jc = jc;
    a.mu0 = mu0;
    a.T = T;
    a.nk02 = 4.0 * (g.nbk - 1) * (g.nbk - 1);
    a.wc = wc;
    a.partial = rs.partial;
    a.bar = rs.bar + 4;
    a.err = reinterpret_cast<int *>(rs.bar + 6);
    a.out = rs.out;
    a.b = b;
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel((const void *)k_mu_roots, dim3(grid, 1, b.P), dim3(kRootThreads), args, 0, st);
    if (e != cudaSuccess) return e;
    return launched();
}

cudaError_t launch_sumrule_roots(const GridDev &g, const double *chiq, const double *chi0_inf, const double *chi0_inf2,
                                 const double *mom_suf, const double *cmax_suf, const double *tailm, double T,
                                 double n, double nsr, double U, double hi_sp, RootScratch rs, cudaStream_t st,
                                 const double *chi0max, double hi_off, const Bp &b) {
    if (g.nb > kRootMaxNb) return cudaErrorInvalidValue;
    int grid = 0;
    cudaError_t e = root_grid(k_sumrule_roots, &grid, rs.max_blocks);
    if (e != cudaSuccess) return e;
    if (b.P > 1) grid = std::max(1, grid / b.P);
    if (rs.reset_sr) {
        e = b.P > 1 ? cudaMemset2DAsync(rs.bar, (size_t)b.arena, 0, 2 * sizeof(unsigned) + sizeof(int), b.P, st)
                    : cudaMemsetAsync(rs.bar, 0, 2 * sizeof(unsigned) + sizeof(int), st);
        if (e != cudaSuccess) return e;
    }
    SumRootArgs a;
    a.chiq = reinterpret_cast<const double4 *>(chiq);
    a.cinf = chi0_inf;
    a.cinf2 = chi0_inf2;
    a.w16 = g.w16;
    a.tailq = g.tailq;
    a.mom_suf = mom_suf;
    a.cmax_suf = cmax_suf;
    a.tailm = tailm;
    a.nb = g.nb;
    a.nblk = g.n8p / 4;
    a.n8 = g.n8;
    a.T = T;
    a.scale = T / (4.0 * (g.nbk - 1) * (g.nbk - 1));
    a.n = n;
    a.nsr = nsr;
    a.U = U;
    a.hi_sp = hi_sp;
    a.chi0max = chi0max;
    a.hi_off = hi_off;
    a.partial = rs.partial;
    a.bar = rs.bar;
    a.err = reinterpret_cast<int *>(rs.bar + 2);
    a.out = rs.out;
    a.b = b;
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel((const void *)k_sumrule_roots, dim3(grid, 1, b.P), dim3(kRootThreads), args, 0,
                                    st);
    if (e != cudaSuccess) return e;
    return launched();
}

cudaError_t launch_barrier_probe(unsigned *words, int withhold, int *blocks, cudaStream_t st) {
    int grid = 0;
    cudaError_t e = root_grid(k_barrier_probe, &grid, 0);
    if (e != cudaSuccess) return e;
    *blocks = grid;
    if ((e = cudaMemsetAsync(words, 0, 4 * sizeof(unsigned), st)) != cudaSuccess) return e;
    void *args[] = {&words, &withhold};
    e = cudaLaunchCooperativeKernel((const void *)k_barrier_probe, dim3(grid), dim3(kRootThreads), args, 0, st);
    if (e != cudaSuccess) return e;
    return launched();
}

}  // namespace tpsc
