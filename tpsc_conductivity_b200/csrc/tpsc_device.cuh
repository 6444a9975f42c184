// tpsc_device.cuh -- device helpers shared by the kernel translation units
// (tpsc_kernels.cu: chi0, vertex, self-energy, traces; tpsc_cond.cu: the
// current-current correlator).  Everything here is internal to the library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "tpsc_fft.cuh"
#include "tpsc_kernels.cuh"

namespace tpsc {

// counts one (or n) kernel launches for the instrumentation ABI and returns
// the launch status
cudaError_t launched(int n = 1);

// Dynamic shared memory above 48 KB needs the function's opt-in attribute,
// which is process-wide: it is raised once per kernel and device to the
// largest size the device allows and never lowered, so that launches from
// concurrent host threads with different sizes all see a cap they fit under.
cudaError_t smem_optin(const void *fn);

namespace {

constexpr double kPi = 3.141592653589793;  // == acos(-1.0) in double

// point blockIdx.z's copy of a per-point array (see Bp)
template <class T>
__device__ __forceinline__ T *at(T *ptr, long long arena) {
    using Ch = typename std::conditional<std::is_const<T>::value, const char, char>::type;
    return ptr ? reinterpret_cast<T *>(reinterpret_cast<Ch *>(ptr) + (long long)blockIdx.z * arena) : ptr;
}
// the point's scalar `slot`, or v for a plain launch
__device__ __forceinline__ double bpar(const Bp &b, int slot, double v) {
    return b.pp ? at(b.pp, b.arena)[slot] : v;
}
constexpr int kSliceThreads = 352;  // 22 groups of 16: the 65 line pairs of a 129-point pass in 3 rounds
constexpr int kTauThreads = 256;
constexpr int kWarm = 30;  // spline sweep warm-up: carry error <= 0.268^30 < 1e-17

// octant index o = m + l (l + 1) / 2, 0 <= m <= l -> (l, m) without a
// table: 8 o + 1 < 2^24 is exact in float and its square root correctly
// rounded, so the estimate of l is off by at most one and the two checks
// correct it
__device__ __forceinline__ void oct_lm(int o, int &l, int &m) {
    int a = (int)((sqrtf((float)(8 * o + 1)) - 1.0f) * 0.5f);
    if ((a + 1) * (a + 2) / 2 <= o) ++a;
    if (a * (a + 1) / 2 > o) --a;
    l = a;
    m = o - a * (a + 1) / 2;
}

// integer multiplicity weight of octant point (l, m) as in the reference
// loops: `base` halved on the l edges, m edges and the diagonal
__device__ __forceinline__ int oct_weight(int base, int l, int m, int nbk) {
    int w = base;
    if (l == 0 || l == nbk - 1) w /= 2;
    if (m == 0 || m == nbk - 1) w /= 2;
    if (m == l) w /= 2;
    return w;
}

// error-free sum of two doubles (Knuth's TwoSum): a + b = s + e exactly
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
    s = a + b;
    const double bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}

// ---------------------------------------------------------------------------
// compensated (Kahan-Babuska) summation
// ---------------------------------------------------------------------------
struct KSum {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x) {
        const double t = s + x;
        if (fabs(s) >= fabs(x))
            c += (s - t) + x;
        else
            c += (x - t) + s;
        s = t;
    }
    // another compensated sum, by TwoSum
    __device__ __forceinline__ void join(double s2, double c2) {
        double t, r;
        two_sum(s, s2, t, r);
        s = t;
        c += c2 + r;
    }
    // the sums of a segment of W lanes (W a power of two, `lanes` its mask), in its first lane
    template <int W>
    __device__ __forceinline__ void join_lanes(unsigned lanes) {
#pragma unroll
        for (int off = W / 2; off > 0; off >>= 1) {
            const double s2 = __shfl_down_sync(lanes, s, off, W), c2 = __shfl_down_sync(lanes, c, off, W);
            join(s2, c2);
        }
    }
    __device__ __forceinline__ double value() const { return s + c; }
};

// ---------------------------------------------------------------------------
// two-pass reductions: per-block partials, then one block adds them in order
// ---------------------------------------------------------------------------
template <int NV>
__device__ void block_store(double (&v)[NV], double *partial) {
    __shared__ double red[32][NV];
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double x = lane < nw ? red[lane][k] : 0.0;
            for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
            if (lane == 0) partial[k * kMaxBlocks + blockIdx.x] = x;
        }
    }
}

// Sum of the per-block partials in a fixed order: block k adds value k, each
// thread a lane-strided compensated sum, then a shuffle tree per warp and the
// warps' totals in order (deterministic).
constexpr int kFinishThreads = 256;
template <int NV>
__global__ void __launch_bounds__(kFinishThreads) k_finish(const double *partial, int nblocks, double *result,
                                                           double offset0, Bp bp) {
    __shared__ double wsum[kFinishThreads / 32];
    const int k = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    partial = at(partial, bp.arena);
    result = at(result, bp.arena);
    KSum acc;
    for (int b = threadIdx.x; b < nblocks; b += kFinishThreads) acc.add(partial[k * kMaxBlocks + b]);
    double v = acc.value();
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) wsum[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kFinishThreads / 32; ++w) t += wsum[w];
        result[k] = t + (k == 0 ? offset0 : 0.0);
    }
}

__global__ void k_max_finish(const double *partial, int nblocks, double *result, Bp bp) {
    partial = at(partial, bp.arena);
    result = at(result, bp.arena);
    double m = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 32) m = fmax(m, partial[b]);
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    if (threadIdx.x == 0) result[0] = m;
}

template <int NV>
cudaError_t finish(Reduce r, int nblocks, double offset0, cudaStream_t st, const Bp &b = Bp{}) {
    k_finish<NV><<<dim3(NV, 1, b.P), kFinishThreads, 0, st>>>(r.partial, nblocks, r.result, offset0, b);
    return launched();
}

// ---------------------------------------------------------------------------
// slice kernels: shared-memory plan of one nbk x nbk slice + FFT scratch
// ---------------------------------------------------------------------------
// FFT groups of an FP64 slice kernel whose lines go through the plain FFT.  A pass
// transforms (NBK + 1)/2 line pairs, one per group of G threads, and the
// groups' scratch is most of the shared memory, so a block holds the groups
// that a pass can use and no more: a fixed 352 threads left 25% (65 lines) to
// 95% (9 lines) of a block idle in the transforms at one CTA per SM.
template <int NBK>
struct SliceGroups {
    static constexpr int G = FftPlan<2 * (NBK - 1)>::G;
    static constexpr int ngrp = NBK >= 129 ? kSliceThreads / G : (NBK + 1) / 2;
    // groups of a kSliceThreads block: the one- to four-CTA boundary kernels,
    // whose single slice should be done as soon as possible
    static constexpr int wide = kSliceThreads / G;
};

template <int NBK, int NG = SliceGroups<NBK>::ngrp>
struct SliceSmem {
    static constexpr int L = 2 * (NBK - 1);
    static constexpr int G = FftPlan<L>::G;
    static constexpr int NGRP = NG;
    static constexpr size_t slice_bytes = (size_t)NBK * NBK * sizeof(double);
    static constexpr size_t scr_off = (slice_bytes + 15) & ~(size_t)15;
    static constexpr size_t tw_off = scr_off + (size_t)NGRP * padded_len(L) * sizeof(double2);
    // the full L-point twiddle table when it fits behind the slice and the
    // groups' FFT scratch, else the two-level table (2 KB)
    static constexpr bool smem_tw = tw_off + (size_t)L * sizeof(double2) <= 232448;
    static constexpr size_t bytes = tw_off + (smem_tw ? (size_t)L * sizeof(double2) : sizeof(TwoLevelTw));
    static_assert(bytes <= 232448, "slice does not fit in shared memory");
};

template <int NBK>
__device__ __forceinline__ double2 *slice_scratch(double *S) {
    return reinterpret_cast<double2 *>(reinterpret_cast<char *>(S) + SliceSmem<NBK>::scr_off);
}

// The L-point twiddles exp(-2 pi i m / L) staged in shared memory behind the
// FFT scratch -- the full table, or where that does not fit the two-level
// table (entry m = hi[m >> 6] lo[m & 63]); the first __syncthreads of the
// kernel publishes it.
template <int NBK, int NG = SliceGroups<NBK>::ngrp>
__device__ __forceinline__ auto slice_twiddles(double *S, const double2 *__restrict__ tw) {
    constexpr int L = SliceSmem<NBK>::L;
    char *base = reinterpret_cast<char *>(S) + SliceSmem<NBK, NG>::tw_off;
    if constexpr (SliceSmem<NBK, NG>::smem_tw) {
        double2 *t = reinterpret_cast<double2 *>(base);
        for (int i = threadIdx.x; i < L; i += blockDim.x) t[i] = __ldg(&tw[i]);
        return (const double2 *)t;
    } else {
        TwoLevelTw *t = reinterpret_cast<TwoLevelTw *>(base);
        for (int i = threadIdx.x; i < 64; i += blockDim.x) {
            t->hi[i] = 64 * i < L ? __ldg(&tw[64 * i]) : make_double2(1.0, 0.0);
            t->lo[i] = i < L ? __ldg(&tw[i]) : make_double2(1.0, 0.0);
        }
        return (const TwoLevelTw *)t;
    }
}

// Threads, shared memory and CTAs per SM of an FP64 slice kernel, and how its
// lines are transformed: by the symmetric FFT (sym_lines) from 33 lines on, which
// takes 0.6 of the plain one's arithmetic and shared-memory traffic and fits 33
// groups where 22 did (129 lines: 2 rounds of line pairs instead of 3); below, one
// radix-16 pass is all of the transform and symmetry saves nothing.  KEEP: G and
// chi0 up to 65 lines stay on the plain FFT -- the reference's diagnostics
// |Usp - Usp(half grid)| / Usp are ~1e-9, so a rounding of chi0 that differs in
// the last bit moves them by 1e-8 of themselves.  129 lines take the symmetric
// one for the 0.1 ms below: either transform leaves the 256^2 diagnostics
// (against the plain half grid) the same noise, relative errors against 64 bits
// of 9 models 3e-16 to 3.5e-8 with the plain, 3e-16 to 4.7e-8 with the symmetric.
// Plain -> symmetric, one launch: correlator slices (two transforms) 256^2 x 4096
// 3390 -> 2940 us, 128^2 x 2048 184 -> 156; G 256^2 778 -> 687, Sigma 724 -> 630;
// Aslamazov-Larkin q -> r 64^2 x 1024 18.0 -> 14.2 us a frequency.
template <int NBK, bool KEEP = false>
struct SlicePlan {
    static constexpr bool sym = NBK >= (KEEP ? 129 : 33);
    static constexpr int warps = NBK >= 129 ? 11 : NBK == 65 ? 6 : 2;  // of symmetric groups
    static constexpr int G = FftPlan<2 * (NBK - 1)>::G;
    static constexpr int threads = sym ? 32 * warps : NBK == 17 ? 64 : (SliceGroups<NBK>::ngrp * G + 31) / 32 * 32;
    static constexpr int blocks = NBK >= 129 ? 1 : NBK == 65 ? 2 : NBK == 33 ? (sym ? 8 : 4) : 8;
    static constexpr size_t scr_off = SliceSmem<NBK>::scr_off;
    static constexpr size_t sym_scr() {
        using F = SymFft<2 * (NBK - 1) >= 64 ? 2 * (NBK - 1) : 64>;
        return (size_t)warps * F::per_warp * F::len * sizeof(double2);
    }
    static constexpr size_t sym_tw() { return SymFft<2 * (NBK - 1) >= 64 ? 2 * (NBK - 1) : 64>::ntw * sizeof(double2); }
    static constexpr size_t tw_off = sym ? scr_off + sym_scr() : SliceSmem<NBK>::tw_off;
    static constexpr size_t bytes = sym ? tw_off + sym_tw() : SliceSmem<NBK>::bytes;
    static_assert(bytes <= 232448, "slice does not fit in shared memory");
};

// SMs of the current device (148 on a whole B200; 0 on an error)
inline int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
}
// A slice launch that PER blocks of kSliceThreads an SM hold at once, up to 65 lines: its
// time is one slice's, and 352 threads instead of the plan's 64 to 192 shorten the loops
// that fill and store it (the transform has no more groups than line pairs to give it).
// The plan's block -> the wide one, one point: 64^2 x 64 G 11.4 -> 7.5 us (FP32) and 8.6 ->
// 6.3 (FP64), V 8.8 -> 7.7 and 10.0 -> 7.1, chi0 8.5 -> 6.9, Sigma 8.6 -> 7.5; 32^2 x 64
// G 6.7 -> 5.5; 128^2 x 64 G 15.0 -> 11.6.
template <class P, int PER>
struct WidePlan : P {
    static constexpr int threads = kSliceThreads, blocks = PER;
    static_assert(P::threads <= kSliceThreads, "a wide block");
};
// f(plan) with the plan of a launch of `slices` slices
template <int NBK, class P, int PER, class F>
cudaError_t with_plan(long long slices, const F &f) {
    if constexpr (NBK <= 65) {
        if (slices <= (long long)PER * sm_count()) return f(WidePlan<P, PER>{});
    }
    return f(P{});
}

// the twiddles of the plan's transform in shared memory (the first
// __syncthreads of the kernel publishes them)
template <int NBK, bool KEEP = false>
__device__ __forceinline__ auto plan_twiddles(double *S, const double2 *__restrict__ tw) {
    if constexpr (SlicePlan<NBK, KEEP>::sym) {
        using F = SymFft<2 * (NBK - 1)>;
        double2 *t = reinterpret_cast<double2 *>(reinterpret_cast<char *>(S) + SlicePlan<NBK, KEEP>::tw_off);
        for (int i = threadIdx.x; i < F::ntw; i += blockDim.x) t[i] = __ldg(&tw[(i / F::G + 1) * (i % F::G)]);
        return (const double2 *)t;
    } else {
        return slice_twiddles<NBK>(S, tw);
    }
}
template <int NBK, bool KEEP = false, class TW>
__device__ __forceinline__ void plan_dct2(double *S, const TW *tws) {
    if constexpr (SlicePlan<NBK, KEEP>::sym)
        sym_dct2_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    else
        dct2_slice<NBK, SliceGroups<NBK>::ngrp>(S, slice_scratch<NBK>(S), tws);
}
template <int NBK, class TW>
__device__ __forceinline__ void plan_dst_dct(double *S, const TW *tws) {
    if constexpr (SlicePlan<NBK>::sym)
        sym_dst_dct_slice<NBK>(S, slice_scratch<NBK>(S), tws);
    else
        dst_dct_slice<NBK, SliceGroups<NBK>::ngrp>(S, slice_scratch<NBK>(S), tws);
}

// U (3 Usp + Uch) / 8 from the device pair Usc = (Usp, Uch), rounded as the
// host expression is (no contraction into an FMA)
__device__ __forceinline__ double vertex_fact(double U, const double *Usc) {
    return __dmul_rn(U, __dadd_rn(__dmul_rn(3.0, Usc[0]), Usc[1])) / 8.0;
}

// c[a] = cos(pi a t / N), a = 0..R, from c1 = cos(pi t / N) (tw64[t].x of the
// table tw64[m] = exp(-2 pi i m / 2N)) by the Chebyshev recurrence
// c[a + 1] = 2 c1 c[a] - c[a - 1]: one table read for all R + 1 cosines, a
// few ulp for R <= 4
template <int R>
__device__ __forceinline__ void cheb_cos(double c1, double (&c)[R + 1]) {
    c[0] = 1.0;
    if constexpr (R >= 1) c[1] = c1;
#pragma unroll
    for (int a = 2; a <= R; ++a) c[a] = fma(2.0 * c1, c[a - 1], -c[a - 2]);
}

// L2 prefetch by the CTA of [p, p + bytes), one request per 128-byte line,
// every address inside the range
__device__ __forceinline__ void prefetch_l2_range(const void *p, size_t bytes) {
    const char *c = static_cast<const char *>(p);
    for (size_t off = (size_t)threadIdx.x * 128; off < bytes; off += (size_t)blockDim.x * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(c + off));
}
// L2 prefetch by the CTA of row j of a four-column-block array (NJ rows per
// block, nblk blocks): one 32-byte piece per block
__device__ __forceinline__ void prefetch_l2_blockrow(const double *a, int j, int NJ, int nblk) {
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + ((size_t)b * NJ + j) * 4));
}

// CTAs that one launch of `kernel` holds on the GPU at once: a slice kernel's
// CTA j prefetches the inputs of slice j + this, which the same launch reaches
// about one wave later
template <class K>
int resident_ctas(K kernel, int threads, size_t smem) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess) return 0;
    return sm_count() * per;
}

// Fill a symmetric NBK x NBK slice from the octant points: value(o) does all
// global reads of point o and returns its value.  Each thread takes KB points
// at a time and issues all their reads before storing any of them, so that
// KB memory round trips overlap instead of running one after the other.
template <int NBK, int KB = 8, class T, class Value>
__device__ __forceinline__ void fill_octant(T *S, int n8, const Value &value) {
    for (int base = threadIdx.x; base < n8; base += KB * blockDim.x) {
        T v[KB];
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            const int o = base + b * blockDim.x;
            if (o < n8) v[b] = value(o);
        }
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            const int o = base + b * blockDim.x;
            if (o < n8) {
                int l, m;
                oct_lm(o, l, m);
                S[l * NBK + m] = v[b];
                S[m * NBK + l] = v[b];
            }
        }
    }
}

// use(i, load(i)) for the block's i < n, KB points of a thread loaded before the
// first of them is used: a loop of one load and one use each waits a memory
// latency per point (with one CTA per SM half the time of the correlator's 129-
// line slices)
template <int KB, class Load, class Use>
__device__ __forceinline__ void batched(int n, const Load &load, const Use &use) {
    for (int base = threadIdx.x; base < n; base += KB * blockDim.x) {
        decltype(load(0)) v[KB];
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            const int i = base + b * blockDim.x;
            if (i < n) v[b] = load(i);
        }
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            const int i = base + b * blockDim.x;
            if (i < n) use(i, v[b]);
        }
    }
}

// write octant value v of point (l, m) into both triangles of the slice
template <int NBK>
__device__ __forceinline__ void put_sym(double *S, int l, int m, double v) {
    S[l * NBK + m] = v;
    S[m * NBK + l] = v;
}

// ---------------------------------------------------------------------------
// tau kernels: clamped spline along a column, staging
// ---------------------------------------------------------------------------
// Clamped cubic spline through y[0..NJ) on a uniform grid of step h with end
// slopes d0, dN: on exit y holds the node second derivatives M_j.  Solves
//   2 M_0 + M_1 = 6/h ((V_1 - V_0)/h - d0)
//   M_{i-1} + 4 M_i + M_{i+1} = 6/h^2 (V_{i+1} - 2 V_i + V_{i-1})
//   M_{N-1} + 2 M_N = 6/h (dN - (V_N - V_{N-1})/h)
// -- the same interpolant as generique::spline_coeffs_rel
// (src/generique.cpp:214-322), S_j''' = 6 a_j = (M_{j+1} - M_j)/h -- by the
// Thomas algorithm with pivots invp = 1/p_i and multipliers cp_i (cp_N = 0)
// precomputed on the host.  The sweeps are split over TPC threads per column:
// each chunk starts its carry kWarm rows early from zero; the carry decays
// by 1/p_i <= 1/(2+sqrt3) per row, so the truncation error is below 1e-17 of
// the local magnitude.  All threads of the block must call.
// RAW: y already holds the right-hand side (the adjoint of the spline solves
// the same symmetric system); h, d0 and dN are not used.
template <int NC = 4, bool RAW = false>
__device__ void spline_second_derivatives(double *A, int lda, int NJ, double h, const double *d0, const double *dN,
                                          const double *__restrict__ invp, const double *__restrict__ cp) {
    const int TPC = blockDim.x / NC;
    const int c = threadIdx.x / TPC, k = threadIdx.x % TPC;
    double *y = A + c * lda;
    const int C = (NJ + TPC - 1) / TPC;
    const int s = min(k * C, NJ), e = min(s + C, NJ);
    const int N = NJ - 1;
    const double a6 = 6.0 / (h * h), b6 = 6.0 / h, ih = 1.0 / h;
    const double dl = RAW ? 0.0 : d0[c], dr = RAW ? 0.0 : dN[c];
    // interior rows kSplinePivotConst <= i < N share one pivot, 1/p = cp: a
    // register instead of a load in the sweeps' dependent chains
    const double cpiv = N > kSplinePivotConst ? __ldg(&invp[kSplinePivotConst]) : 0.0;
    auto piv = [&](int i) -> double { return (i >= kSplinePivotConst && i < N) ? cpiv : __ldg(&invp[i]); };
    auto sup = [&](int i) -> double { return (i >= kSplinePivotConst && i < N) ? cpiv : __ldg(&cp[i]); };
    auto rhs = [&](int i, double vm, double v0, double vp) -> double {
        if (RAW) return v0;
        if (i == 0) return b6 * ((vp - v0) * ih - dl);
        if (i == N) return b6 * (dr - (v0 - vm) * ih);
        return a6 * (vp - 2.0 * v0 + vm);
    };
    double carry = 0.0, vm_h = 0.0, vs_h = 0.0, ve_h = 0.0;
    if (s < e) {
        if (s > 0) {
            const int i0 = max(0, s - kWarm);
            double cc = 0.0;
            double vm = i0 > 0 ? y[i0 - 1] : 0.0, v0 = y[i0];
            for (int i = i0; i < s; ++i) {
                const double vp = y[i + 1];
                cc = (rhs(i, vm, v0, vp) - cc) * piv(i);
                vm = v0;
                v0 = vp;
            }
            carry = cc;
            vm_h = y[s - 1];
        }
        vs_h = y[s];
        ve_h = e < NJ ? y[e] : 0.0;
    }
    __syncthreads();
    if (s < e) {
        double vm = vm_h, v0 = vs_h;
        for (int i = s; i < e; ++i) {
            const double vp = (i + 1 < e) ? y[i + 1] : ve_h;
            const double dp = (rhs(i, vm, v0, vp) - carry) * piv(i);
            y[i] = dp;
            carry = dp;
            vm = v0;
            v0 = vp;
        }
    }
    __syncthreads();
    double mc = 0.0;
    if (s < e && e < NJ) {
        const int i1 = min(N, e - 1 + kWarm);
        double mm = 0.0;
        for (int i = i1; i >= e; --i) mm = y[i] - sup(i) * mm;
        mc = mm;
    }
    __syncthreads();
    if (s < e) {
        double mm = mc;
        for (int i = e - 1; i >= s; --i) {
            mm = y[i] - sup(i) * mm;
            y[i] = mm;
        }
    }
    __syncthreads();
}

// per-column sum of y[i0..i1) over the TPC threads of each column -> out[c]:
// compensated per-thread sums, then a fixed shuffle tree that adds the pairs
// (sum, compensation) with TwoSum, then the column's warps in order.  TPC is
// a multiple of 32 (blockDim.x = 32 NC k).
template <int NC = 4>
__device__ void column_sums(const double *A, int lda, int i0, int i1, double *out) {
    const int TPC = blockDim.x / NC;
    const int c = threadIdx.x / TPC, k = threadIdx.x % TPC;
    KSum acc;
    for (int i = i0 + k; i < i1; i += TPC) acc.add(A[c * lda + i]);
    acc.join_lanes<32>(0xffffffffu);
    __shared__ double2 part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_double2(acc.s, acc.c);
    __syncthreads();
    if (k == 0) {
        const int w0 = threadIdx.x >> 5, nw = TPC >> 5;
        for (int q = 1; q < nw; ++q) acc.join(part[w0 + q].x, part[w0 + q].y);
        out[c] = acc.value();
    }
    __syncthreads();
}

template <int N>
struct TauSmem {
    static constexpr int threads = (N / 16) > kTauThreads ? (N / 16) : kTauThreads;
    // four staged columns, the FFT scratch, then the two-level twiddle tables
    __host__ __device__ static size_t tables_off(int NJ) {
        return (((size_t)4 * NJ * sizeof(double) + 15) & ~(size_t)15) + (size_t)padded_len(N) * sizeof(double2);
    }
    __host__ __device__ static size_t bytes(int NJ) { return tables_off(NJ) + 2 * sizeof(TwoLevelTw); }
};

// Two-level tables (shared memory) of the N-point FFT twiddles tw[m] =
// exp(-2 pi i m/N) and of the pre-twiddles ht[m] = exp(+i pi m/N), m < N,
// from the global tables; entry m is hi[m >> 6] * lo[m & 63].  The caller's
// next barrier publishes them.
__device__ __forceinline__ void tau_tables(TwoLevelTw *tw2, TwoLevelTw *ht2, const double2 *__restrict__ tw,
                                           const double2 *__restrict__ ht, int N) {
    for (int t = threadIdx.x; t < 64; t += blockDim.x) {
        const double2 one = make_double2(1.0, 0.0);
        tw2->hi[t] = 64 * t < N ? __ldg(&tw[64 * t]) : one;
        tw2->lo[t] = t < N ? __ldg(&tw[t]) : one;
        ht2->hi[t] = 64 * t < N ? __ldg(&ht[64 * t]) : one;
        ht2->lo[t] = t < N ? __ldg(&ht[t]) : one;
    }
}
__device__ __forceinline__ double2 tw_at(const TwoLevelTw *t, int m) { return cmul(t->hi[m >> 6], t->lo[m & 63]); }

// Asynchronous 8-byte global -> shared copy (cp.async); the issuing thread
// waits for its own copies with cp_async_wait_all, a barrier then publishes
// them.  A thread keeps all its copies in flight at once, which is what
// streams a column block in at HBM speed with one CTA per SM.
__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
// input staging of the slice kernels whose inputs are rows of global arrays:
// the slice and the FFT scratch are idle until the fill, so a CTA first copies
// its input rows there with asynchronous copies (all in flight at once: one
// memory latency per slice instead of one per batch of loads), waits for its
// own copies, and forms the slice from shared memory
// ---------------------------------------------------------------------------
template <int NBK>
struct StageRows {
    static constexpr int N8 = NBK * (NBK + 1) / 2;
    static constexpr int N8P = (N8 + 3) & ~3;
    static constexpr size_t blockrow_bytes = (size_t)N8P * sizeof(double);  // one row of a column-block array
    static constexpr size_t drow_bytes = ((size_t)N8 * sizeof(double) + 15) & ~(size_t)15;  // one FP64 row
};

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// row j of a column-block array a (NJ rows) -> dst[o], o < N8P (16-byte copies)
template <int NBK>
__device__ __forceinline__ void stage_blockrow(double *dst, const double *__restrict__ a, int j, int NJ) {
    for (int i = threadIdx.x; i < StageRows<NBK>::N8P / 2; i += blockDim.x) {
        const int b = i >> 1, h = i & 1;
        cp_async16(dst + 4 * b + 2 * h, a + ((size_t)b * NJ + j) * 4 + 2 * h);
    }
}
// n8 doubles from src -> dst (8-byte copies: rows of an [j][o] array are
// 16-byte aligned only for even j)
template <int NBK>
__device__ __forceinline__ void stage_drow(double *dst, const double *__restrict__ src) {
    for (int o = threadIdx.x; o < StageRows<NBK>::N8; o += blockDim.x) cp_async8(dst + o, src + o);
}
// Form the symmetric slice from value(o), which reads the staged inputs:
// every thread computes its octant points into registers, then a barrier (the
// staging area overlaps the slice), then the writes of both triangles.
// THREADS: the block size the kernel is launched with.
template <int NBK, int THREADS, class T, class Value>
__device__ __forceinline__ void fill_from_staged(T *S, const Value &value) {
    constexpr int N8 = StageRows<NBK>::N8, PER = (N8 + THREADS - 1) / THREADS;
    T v[PER];
#pragma unroll
    for (int b = 0; b < PER; ++b) {
        const int o = threadIdx.x + b * THREADS;
        if (o < N8) v[b] = value(o);
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < PER; ++b) {
        const int o = threadIdx.x + b * THREADS;
        if (o < N8) {
            int l, m;
            oct_lm(o, l, m);
            S[l * NBK + m] = v[b];
            S[m * NBK + l] = v[b];
        }
    }
}


// Load one column block into shared memory, column-major (the caller's next
// __syncthreads publishes it).  Padding columns (octant index >= n8, present
// because N8 is rounded up to a multiple of 4) load as zeros: they share
// packed FFTs with real columns, so stale values there would leak into real
// outputs through rounding.
__device__ __forceinline__ void stage_in(double *A, const double *g, int NJ, int nvalid) {
    for (int i = threadIdx.x; i < 4 * NJ; i += blockDim.x) {
        double *dst = &A[(i & 3) * NJ + (i >> 2)];
        if ((i & 3) < nvalid)
            cp_async8(dst, g + i);
        else
            *dst = 0.0;
    }
    cp_async_wait_all();
}
__device__ __forceinline__ void stage_out(const double *A, double *g, int NJ) {
    for (int i = threadIdx.x; i < 4 * NJ; i += blockDim.x) g[i] = A[(i & 3) * NJ + (i >> 2)];
}

// full Sigma(k, i w_n) = Sinf/z + C2/z^2 + C3/z^3 + S/z^4, z = i w_n, from the
// reciprocal powers of w_n
__device__ __forceinline__ void sigma_full(double i1, double sinf, double c2, double c3, double2 Sv, double &rS,
                                           double &iS) {
    const double i2 = i1 * i1, i4 = i2 * i2;
    rS = -c2 * i2 + Sv.x * i4;
    iS = -sinf * i1 + c3 * i2 * i1 + Sv.y * i4;
}

// The sum rules' Matsubara tail: with x_n = 1/qn^2, chi_n = a x_n + b x_n^2 and h = sgn U/2,
//   chi/(1 + h chi) - chi = sum_{m>=1} (-h)^m chi^{m+1},
//   sum_n chi_n^{m+1} = sum_i C(m+1, i) a^{m+1-i} b^i Q_{m+1+i},
// with the U-independent power sums Q_k = sum_n x_n^k (tailq[k], k <= 2 kTailM + 2).
// A column whose |h chi_max| >= kTailSeriesMax is summed term by term.
constexpr int kTailM = 8;
constexpr double kTailSeriesMax = 0.004;  // (0.004)^8 < 1e-19: series truncation below rounding

// the power sums S_{m+1} = sum_n chi_n^{m+1}, m = 1..kTailM, of one column
__device__ __forceinline__ void tail_sums(double a, double b, const double *__restrict__ Q, double (&S)[kTailM]) {
    double ap[kTailM + 2], bp[kTailM + 2];
    ap[0] = bp[0] = 1.0;
#pragma unroll
    for (int k = 1; k < kTailM + 2; ++k) {
        ap[k] = ap[k - 1] * a;
        bp[k] = bp[k - 1] * b;
    }
#pragma unroll
    for (int m = 1; m <= kTailM; ++m) {
        const int p = m + 1;
        double Sp = 0.0, coef = 1.0;  // coef = C(p, i)
#pragma unroll
        for (int i = 0; i <= p; ++i) {
            Sp += coef * ap[p - i] * bp[i] * __ldg(&Q[p + i]);
            coef = coef * (p - i) / (i + 1);
        }
        S[m - 1] = Sp;
    }
}

__device__ __forceinline__ void tail_series(double a, double b, double h, const double *__restrict__ Q, double &f,
                                           double &dfdh) {
    double S[kTailM];
    tail_sums(a, b, Q, S);
    f = 0.0;
    dfdh = 0.0;
    double hm = 1.0;  // (-h)^(m-1)
#pragma unroll
    for (int m = 1; m <= kTailM; ++m) {
        f += (-h) * hm * S[m - 1];     // (-h)^m S_p
        dfdh += -m * hm * S[m - 1];    // d/dh (-h)^m = -m (-h)^(m-1)
        hm *= -h;
    }
}

// 32-byte streaming load (two 16-byte evict-first loads)
__device__ __forceinline__ double4 ld_stream4(const double4 *p) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    const double2 a = __ldcs(q), b = __ldcs(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// one term of Tr(G - G0) (green::traceDiffG, src/green.cpp:3108-3182) and its
// derivative with respect to the chemical potential pmu: w Re[G - G0] with
// G = 1/(i w_n - e + pmu - Sigma), G0 = 1/(i w_n - e + mu0).  The value's products are
// fused here, not by the compiler, which does it by what stands beside them: find_zero
// ends at the last bits of the sum, and a search on the host then took other steps (9
// evaluations for 20) than the device's.
__device__ __forceinline__ void trdiff_term(double wn, double rS, double iS, double e, double mu0, double pmu,
                                            double w, double &v, double &dv) {
    const double a = e - pmu + rS, d = e - mu0, g = mu0 - pmu + rS, y = wn - iS, wn2 = __dmul_rn(wn, wn);
    const double A2 = fma(y, y, __dmul_rn(a, a));
    const double num = fma(-wn2, g, fma(__dmul_rn(g, a), d, __dmul_rn(__dmul_rn(iS, fma(-2.0, wn, iS)), d)));
    const double inv = w / __dmul_rn(A2, fma(d, d, wn2));
    v = fma(inv, num, v);
    dv += inv * (wn * wn - (a + g) * d + num * 2.0 * a / A2);
}
// the same with the second derivative: d2/dpmu2 w Re G = 2 w Re G^3, and
// with z = x + i y (x = -a, y = w_n - Im Sigma), Re conj(z)^3 = x^3 - 3 x y^2
__device__ __forceinline__ void trdiff_term(double wn, double rS, double iS, double e, double mu0, double pmu,
                                            double w, double &v, double &dv, double &d2v) {
    trdiff_term(wn, rS, iS, e, mu0, pmu, w, v, dv);
    const double x = pmu - e - rS, y = wn - iS, r = 1.0 / (x * x + y * y);
    d2v += 2.0 * w * x * (x * x - 3.0 * y * y) * (r * r * r);
}

// Sigma in those terms: as sigma_full, and its asymptotic tail, rounded the same way
// wherever they are formed
__device__ __forceinline__ void trdiff_sigma(double i1, double sinf, double c2, double c3, double2 Sv, double &rS,
                                             double &iS) {
    const double i2 = __dmul_rn(i1, i1), i4 = __dmul_rn(i2, i2);
    rS = fma(Sv.x, i4, -__dmul_rn(c2, i2));
    iS = fma(Sv.y, i4, fma(__dmul_rn(c3, i2), i1, -__dmul_rn(sinf, i1)));
}
__device__ __forceinline__ void trdiff_sigma_tail(double i1, double sinf, double c2, double c3, double c4, double &rS,
                                                  double &iS) {
    const double i2 = __dmul_rn(i1, i1);
    rS = fma(__dmul_rn(c4, i2), i2, -__dmul_rn(c2, i2));
    iS = fma(__dmul_rn(c3, i2), i1, -__dmul_rn(sinf, i1));
}

// a row of four: streamed (read once), or left in the caches for the next pass
template <bool STREAM>
__device__ __forceinline__ double4 ld_row(const double4 *p) {
    return STREAM ? ld_stream4(p) : *p;
}

// a thread's share of column block blk of the sum-rule trace and of its U
// derivative (k_sumrule; the reference form's root search takes the same
// values in the same order): the stored frequencies j < jdir, ww the block's
// weights, and the tail n = nwmax+1 .. 2 nwmax, S(c, f, dfdh) the series of column c
template <bool STREAM>
__device__ __forceinline__ void sumrule_stored(const double4 *__restrict__ chiq, const double (&ww)[4], int blk, int nb,
                                               int jdir, double hu, double &v, double &dv) {
    v = dv = 0.0;
    const double4 *col = chiq + (size_t)blk * nb;
#pragma unroll STREAM ? 1 : 4
    for (int j = threadIdx.x; j < jdir; j += blockDim.x) {
        const double4 x = ld_row<STREAM>(&col[j]);
        const double f = j == 0 ? 0.5 : 1.0;
        const double xs[4] = {x.x, x.y, x.z, x.w};
        double sv = 0.0, sd = 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double q = xs[c] / (1.0 + hu * xs[c]);
            sv += ww[c] * (q - xs[c]);
            sd += ww[c] * q * q;
        }
        v += f * sv;
        dv += f * sd;
    }
}
template <class Series>
__device__ __forceinline__ void sumrule_tail(const double *__restrict__ cinf, const double *__restrict__ cinf2,
                                             const double (&ww)[4], int blk, int nb, double hu, double sgn, double T,
                                             double &tv, double &tdv, const Series &series) {
    tv = tdv = 0.0;
    const int nwmax = nb - 1, o0 = 4 * blk;
    const double tw = 2.0 * 3.141592653589793 * T;
    const double wn1 = (nwmax + 1) * tw;
    const double x1 = 1.0 / (wn1 * wn1);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (ww[c] == 0.0) continue;
        const double a = cinf[o0 + c], b = cinf2[o0 + c];
        const double cmax = fabs(a) * x1 + fabs(b) * x1 * x1;
        if (fabs(hu) * cmax < kTailSeriesMax) {
            if (threadIdx.x == c) {
                double f, dfdh;
                series(c, a, b, f, dfdh);
                tv += ww[c] * f;
                tdv += ww[c] * dfdh * (0.5 * sgn);
            }
        } else {
            for (int t = threadIdx.x; t < nwmax; t += blockDim.x) {
                const double wn = (nwmax + 1 + t) * tw;
                const double i2 = 1.0 / (wn * wn);
                const double xv = a * i2 + b * i2 * i2;
                const double q = xv / (1.0 + hu * xv);
                tv += ww[c] * (q - xv);
                tdv += ww[c] * (-0.5 * sgn) * q * q;
            }
        }
    }
}

// a thread's share of column block blk of Tr(G - G0) at pmu and of its
// derivative (k_trace_diff_G and the reference form's root search)
template <bool STREAM>
__device__ __forceinline__ void trace_diff_block(const double2 *__restrict__ S, const double *__restrict__ s2,
                                                 const double *__restrict__ s3, const double *__restrict__ s4,
                                                 const double *__restrict__ sinfp, const double *__restrict__ ek,
                                                 const double *__restrict__ w16, int blk, int nw0, double mu0,
                                                 double pmu, double T, int jdir, int tail, double &v, double &dv) {
    const int NO = nw0 / 2;
    const double sinf = sinfp[0];
    v = dv = 0.0;
    const int o0 = 4 * blk;
    double ww[4], e[4], c2[4], c3[4], c4[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        ww[c] = w16[o0 + c];
        const bool ok = ww[c] != 0.0;
        e[c] = ok ? ek[o0 + c] : 0.0;
        c2[c] = ok ? s2[o0 + c] : 0.0;
        c3[c] = ok ? s3[o0 + c] : 0.0;
        c4[c] = ok ? s4[o0 + c] : 0.0;
    }
    const double pt = 3.141592653589793 * T;
    const double4 *row = reinterpret_cast<const double4 *>(S + (size_t)blk * 4 * NO);
    for (int j = threadIdx.x; j < jdir; j += blockDim.x) {
        const double wn = __dmul_rn(2 * j + 1, pt);
        const double i1 = 1.0 / wn;
        const double4 p = ld_row<STREAM>(&row[2 * j]), q = ld_row<STREAM>(&row[2 * j + 1]);
        const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                               make_double2(q.z, q.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (ww[c] == 0.0) continue;
            double rS, iS;
            trdiff_sigma(i1, sinf, c2[c], c3[c], sv[c], rS, iS);
            trdiff_term(wn, rS, iS, e[c], mu0, pmu, ww[c], v, dv);
        }
    }
    for (int t = threadIdx.x; tail && t <= NO; t += blockDim.x) {
        const int j = NO + t;
        const double wn = __dmul_rn(2 * j + 1, pt);
        const double i1 = 1.0 / wn;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (ww[c] == 0.0) continue;
            double rS, iS;
            trdiff_sigma_tail(i1, sinf, c2[c], c3[c], c4[c], rS, iS);
            trdiff_term(wn, rS, iS, e[c], mu0, pmu, ww[c], v, dv);
        }
    }
}

// a thread's share of column block blk of green::traceSelfG2 at mu
// (src/green.cpp:2929-2976)
template <bool STREAM>
__device__ __forceinline__ double trace_self2_block(const double2 *__restrict__ S, const double *__restrict__ s2,
                                                    const double *__restrict__ s3, const double *__restrict__ sinfp,
                                                    const double *__restrict__ ek, const double *__restrict__ w16,
                                                    int blk, int nw0, double mu, double T, double nk02) {
    const int o0 = 4 * blk, NO = nw0 / 2;
    const double sinf = sinfp[0];
    const double pt = 3.141592653589793 * T;
    KSum v;
    const double4 *row = reinterpret_cast<const double4 *>(S + (size_t)blk * 4 * NO);
    for (int j = threadIdx.x; j < NO; j += blockDim.x) {
        const double wn = (2 * j + 1) * pt;
        const double i1 = 1.0 / wn;
        const double4 p = ld_row<STREAM>(&row[2 * j]), q = ld_row<STREAM>(&row[2 * j + 1]);
        const double2 sv[4] = {make_double2(p.x, p.y), make_double2(p.z, p.w), make_double2(q.x, q.y),
                               make_double2(q.z, q.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double w8 = 0.5 * w16[o0 + c];
            if (w8 == 0.0) continue;
            double rS, iS;
            sigma_full(i1, sinf, s2[o0 + c], s3[o0 + c], sv[c], rS, iS);
            const double a = ek[o0 + c] - mu + rS;
            const double tmp = w8 * T * 2 / (nk02 * ((wn - iS) * (wn - iS) + a * a));
            v.add(tmp * (iS * wn - iS * iS - (ek[o0 + c] - mu) * rS - rS * rS));
        }
    }
    return v.value();
}

// complex division
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
    // Smith's algorithm
    if (fabs(b.x) >= fabs(b.y)) {
        const double r = b.y / b.x, d = b.x + b.y * r;
        return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
    } else {
        const double r = b.x / b.y, d = b.y + b.x * r;
        return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
    }
}

// ---------------------------------------------------------------------------
// helpers of the current-current correlator kernels (tpsc_cond.cu, tpsc_al.cu)
// ---------------------------------------------------------------------------
// two-column-block layout of the h V and f0 V tau arrays: element (j, c)
__host__ __device__ __forceinline__ size_t bidx2(int j, int c, int NJ) {
    return ((size_t)(c >> 1) * NJ + j) * 2 + (c & 1);
}

// octant index of lattice point (x, y), 0 <= x, y < nbk
__device__ __forceinline__ int oct_index(int x, int y) {
    const int a = max(x, y), b = min(x, y);
    return b + a * (a + 1) / 2;
}

__device__ __forceinline__ double2 cexp2(double2 z) {
    const double ea = exp(z.x);
    if (z.y == 0.0) return make_double2(ea, 0.0);
    double s, c;
    sincos(z.y, &s, &c);
    return make_double2(ea * c, ea * s);
}

__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// T / z by one division
__device__ __forceinline__ double2 crecip(double T, double x, double y) {
    const double s = T / (x * x + y * y);
    return make_double2(x * s, -y * s);
}

// block-wide sum of NV values per thread -> out[0..NV) (all threads must call;
// out visible to every thread on return)
template <int NV>
__device__ void block_sum(double (&v)[NV], double *out) {
    __shared__ double red[32][NV];
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x < NV) {
        const int nw = (blockDim.x + 31) >> 5;
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += red[w][threadIdx.x];
        out[threadIdx.x] = s;
    }
    __syncthreads();
}
// block_sum of compensated sums: the compensations are carried through the tree (a
// plain tree after compensated threads rounds once per level)
template <int NV>
__device__ void block_ksum(KSum (&v)[NV], double *out) {
    __shared__ double2 red[32][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        v[k].template join_lanes<32>(0xffffffffu);
        if (lane == 0) red[warp][k] = make_double2(v[k].s, v[k].c);
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        const int nw = (blockDim.x + 31) >> 5;
        KSum a;
        for (int w = 0; w < nw; ++w) a.join(red[w][threadIdx.x].x, red[w][threadIdx.x].y);
        out[threadIdx.x] = a.value();
    }
    __syncthreads();
}

// split of a packed FFT of two real sequences at bins n and N - n
__device__ __forceinline__ void split_real(double2 Z, double2 Zc, double2 &Fa, double2 &Fb) {
    Fa = make_double2(0.5 * (Z.x + Zc.x), 0.5 * (Z.y - Zc.y));
    Fb = make_double2(0.5 * (Z.y + Zc.y), -0.5 * (Z.x - Zc.x));
}

// Stage the two columns of pair p (contiguous in the two-column-block layout)
// column-major into R; a padding column loads zeros.
__device__ __forceinline__ void stage_pair(double *R, const double *g, int NJ, bool two) {
    for (int i = threadIdx.x; i < 2 * NJ; i += blockDim.x) {
        double *dst = &R[(i & 1) * NJ + (i >> 1)];
        if ((i & 1) && !two)
            *dst = 0.0;
        else
            cp_async8(dst, g + i);
    }
    cp_async_wait_all();
}

// The clamped spline's sweeps for one complex column (or two real ones as its
// parts) of NJ <= N + 1 nodes in the padded layout, in place, by the G threads of
// a group of the N-point FFT: both parts of a node by one thread, so that its two
// chains interleave.  TPC of them sweep, in chunks long enough that the kWarm
// warm-up rows do not dominate.  rhs(i, X[i-1], X[i], X[i+1]) is row i of the
// right-hand side (the neighbour beyond an end is not to be used).
template <int N, class Rhs>
__device__ void spline_sweeps(double2 *X, int NJ, int t, int grp, const double *__restrict__ invp,
                              const double *__restrict__ cp, const Rhs &rhs) {
    constexpr int G = FftPlan<N>::G, TPC = G >= 64 ? G / 2 : G;
    const int C = (NJ + TPC - 1) / TPC, last = NJ - 1;
    const int s = t < TPC ? min(t * C, NJ) : NJ, e = min(s + C, NJ);
    const double cpiv = last > kSplinePivotConst ? __ldg(&invp[kSplinePivotConst]) : 0.0;
    auto piv = [&](int i) -> double { return (i >= kSplinePivotConst && i < last) ? cpiv : __ldg(&invp[i]); };
    auto sup = [&](int i) -> double { return (i >= kSplinePivotConst && i < last) ? cpiv : __ldg(&cp[i]); };
    const double2 zero = make_double2(0.0, 0.0);
    double2 carry = zero, vm_h = zero, vs_h = zero, ve_h = zero;
    if (s < e) {
        if (s > 0) {
            const int i0 = max(0, s - kWarm);
            double2 vm = i0 > 0 ? X[pidx(i0 - 1)] : zero, v0 = X[pidx(i0)];
            for (int i = i0; i < s; ++i) {
                const double2 vp = X[pidx(i + 1)];
                carry = cscale(csub(rhs(i, vm, v0, vp), carry), piv(i));
                vm = v0;
                v0 = vp;
            }
            vm_h = X[pidx(s - 1)];
        }
        vs_h = X[pidx(s)];
        if (e < NJ) ve_h = X[pidx(e)];
    }
    group_sync<G>(grp);
    if (s < e) {
        double2 vm = vm_h, v0 = vs_h;
        for (int i = s; i < e; ++i) {
            const double2 vp = (i + 1 < e) ? X[pidx(i + 1)] : ve_h;
            carry = cscale(csub(rhs(i, vm, v0, vp), carry), piv(i));
            X[pidx(i)] = carry;
            vm = v0;
            v0 = vp;
        }
    }
    group_sync<G>(grp);
    double2 mm = zero;
    if (s < e && e < NJ)
        for (int i = min(last, e - 1 + kWarm); i >= e; --i) mm = csub(X[pidx(i)], cscale(mm, sup(i)));
    group_sync<G>(grp);
    if (s < e)
        for (int i = e - 1; i >= s; --i) {
            mm = csub(X[pidx(i)], cscale(mm, sup(i)));
            X[pidx(i)] = mm;
        }
    group_sync<G>(grp);
}

// spline_second_derivatives for such a column: the node values in X become the
// node second derivatives
template <int N>
__device__ void spline_complex(double2 *X, int NJ, int t, int grp, double h, double2 d0, double2 dN,
                               const double *__restrict__ invp, const double *__restrict__ cp) {
    const int last = NJ - 1;
    const double a6 = 6.0 / (h * h), b6 = 6.0 / h, ih = 1.0 / h;
    auto rhs1 = [&](int i, double vm, double v0, double vp, double dl, double dr) -> double {
        if (i == 0) return b6 * ((vp - v0) * ih - dl);
        if (i == last) return b6 * (dr - (v0 - vm) * ih);
        return a6 * (vp - 2.0 * v0 + vm);
    };
    spline_sweeps<N>(X, NJ, t, grp, invp, cp, [&](int i, double2 vm, double2 v0, double2 vp) -> double2 {
        return make_double2(rhs1(i, vm.x, v0.x, vp.x, d0.x, dN.x), rhs1(i, vm.y, v0.y, vp.y, d0.y, dN.y));
    });
}

// ---------------------------------------------------------------------------
// dispatch over the compiled sizes
// ---------------------------------------------------------------------------
template <template <int> class F, typename... Args>
cudaError_t dispatch_nbk(int nbk, Args... args) {
    switch (nbk) {
        case 5: return F<5>::run(args...);
        case 9: return F<9>::run(args...);
        case 17: return F<17>::run(args...);
        case 33: return F<33>::run(args...);
        case 65: return F<65>::run(args...);
        case 129: return F<129>::run(args...);
        default: return cudaErrorInvalidValue;
    }
}
template <template <int> class F, typename... Args>
cudaError_t dispatch_nw(int nw0, Args... args) {
    switch (nw0) {
        case 16: return F<16>::run(args...);
        case 32: return F<32>::run(args...);
        case 64: return F<64>::run(args...);
        case 128: return F<128>::run(args...);
        case 256: return F<256>::run(args...);
        case 512: return F<512>::run(args...);
        case 1024: return F<1024>::run(args...);
        case 2048: return F<2048>::run(args...);
        case 4096: return F<4096>::run(args...);
        default: return cudaErrorInvalidValue;
    }
}

template <typename K>
cudaError_t set_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return smem_optin((const void *)kernel);
}

}  // namespace
}  // namespace tpsc
