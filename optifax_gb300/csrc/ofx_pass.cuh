// ofx_pass.cuh -- the persistent crystal-pass kernel.
//
// One thread-block cluster of C CTAs propagates one pulse of N = C * M points
// through the whole crystal in a single launch.  CTA rank c holds time points
// n1 M + n2, n1 < C, for the M/C values n2 of its columns [c M/C, (c+1) M/C): C
// segments of M/C consecutive points.  So the C-point DFTs over n1, the first step of
// the four-step transform, are local, the inverse ends where the next step begins, and
// only the two middle exchanges of a transform pair cross the cluster; the stencil pays
// for it with a halo at both ends of every segment.  After the forward transform the
// CTA holds the spectral modes k = c + C k2 (k2 = 0..M-1).  Thread t owns P consecutive
// time points, the local ones P t .. P t + P-1 (held in registers across steps), and
// spectral slots P t .. P t + P-1 (mode k2 = bitrev(slot)).
//
// Per step attempt (reference: OPO_CUDA_BATCH_XTAL.cu:432-506, Heun;
// ode23/OPO_CUDA_ODE23.cu:446-538, RK23):
//   RK stages: NL drive (A^2 e^{i phi} + 2|A|^2 e^{-i phi}, phi = w0 t - bdiffw0 z),
//   shock-term central difference, stage combine -- all in registers, with
//   the +-1 neighbours exchanged by shuffles and shared memory.  Error
//   classification (max-norm, percent) is an OR-reduction over the pulse (or over
//   the batch when the reference's shared schedule is requested).  Accepted steps
//   run the absorber, the forward FFT, the dispersion multiply, the inverse FFT and
//   the 1/N scale without leaving the SM (cluster exchange for C > 1).
//
// Precision: FP32 field and FFT; phases exact in 64-bit fixed point (time
// carrier w0 t, z carrier bdiffw0 z, accumulated dispersion beta z).  The
// linear sub-step is applied as an increment, A_new = E + IFFT((D-1) FFT(E))/N,
// with D - 1 = -2 sin^2(beta s/2) - i sin(beta s) evaluated without
// cancellation, so transform rounding scales with |D - 1| rather than |E|; the
// per-mode phase of every step is the exact fixed-point one of its position (no
// drift of the accumulated phase); the inverse FFT applies the exact reciprocal of
// each forward twiddle.
//
// What bounds it: instruction issue and latency on one SM per 4096 points; HBM is
// idle by design.  Hence packed FP32 pairs, eight points per thread (four below 2048
// points per CTA) for 16 warps where 2048 or more points share a CTA, every table in
// shared memory, and square roots off the common path of the error class.
#pragma once
#include <cooperative_groups.h>
#include "ofx_fft.cuh"
#include "../../include/optifax.h"

namespace cg = cooperative_groups;

namespace ofx {

enum { TIME_SHIFTED = 0, TIME_UNSHIFTED = 1, TIME_NEE = 2 };
enum { ABC_SOFT = 0, ABC_NONE = 1, ABC_HARD = 2, ABC_NEE = 3 };

struct PulseDev {
    const float2* E_in;
    float2* A_out;
    const float* alpha;
    const float* beta;
    const float* G;
    float2* Ap;
    float* stepmods;
    int* trace;
    const int* forced;
    optifax_pulse_stats* stats;
    double bdiffw0, dt;
    uint64_t tau_theta;      // w0 dt in turns (fixed point)
    uint64_t tau_z4;         // bdiffw0 h / 4 in turns (fixed point), per quarter step
    float w0, h, max_err, min_err, sel, c_shock;
    int N, S, nchunks, stepmods_limit, trace_cap, n_forced;
    // synchronously pumped OPO (fb != nullptr): per-mode round-trip transfer
    const float2* fb;        // crystal-output spectrum -> next crystal-input spectrum
    const float2* pump;      // pump spectrum added at the crystal input each trip
    const float* tally_w;    // n_tally x N energy weights on the crystal-output spectrum
    optifax_trip_record* trips;
    int n_trips, n_tally, steady_trips, steady_tally;
    float steady_tol;
    float2* hist;            // optional per-trip crystal-output spectra (n_trips x N)
    const float* esd_w;      // n_esd x N spectral-energy weights (trip sums into esd)
    float* esd;
    int n_esd;
    float* smt;              // optional per-trip stepmods records (n_trips x S)
    float2* xs;              // cavities: the trip's crystal output (N), scratch of the cavity step
};

// Global tables from which every CTA fills its shared-memory ones:
// W_M^x from the quarter period, W_N^e = W_M^{(64/C)(e >> 6)} W_N^{e & 63}
struct FftTables {
    const Twiddle* quad;     // W_M^y, y in [0, M/4)
    const Twiddle* low;      // W_N^i, i in [0, 64)
};

struct KernelCfg {
    int time_mode;
    int abc_mode;
    int guard;           // XTAL/BATCH_OP: ceil chunk count and k < Nsteps loop guard
    int shared_sched;    // 1: OR the error flags over every pulse of the launch (grid barrier)
    int max_attempts_mul;
    unsigned long long* grid_sync;   // shared schedule: 4 words, zero before the launch; the last: a wait ran out
    int clusters;        // of the launch
    int wait;            // limit of a bounded wait, in looks at an mbarrier (about 4 us each)
};
constexpr int kWait = 1 << 19;       // about 2 s

// Kernel flavours: the MEX Heun and RK23 schedules (OPTIFAX_HEUN, OPTIFAX_RK23) and
// the Heun schedule with NEE_CPU.m step control, a separate instantiation so the
// MEX kernels carry no NEE branches.
constexpr int kHeunNee = 2;

// ---------------------------------------------------------------------------
// pointwise physics
// ---------------------------------------------------------------------------
// Pairs of points (j, j + P/2) of one thread in structure-of-arrays form: `re` and
// `im` hold the two points' parts, so that every operation of the stages is packed.
struct Pair { float2 re, im; };

__device__ __forceinline__ Pair pair_add(const Pair& a, const Pair& b) { return Pair{add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Pair pair_sub(const Pair& a, const Pair& b) { return Pair{sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a s + b
__device__ __forceinline__ Pair pair_fma(const Pair& a, float s, const Pair& b) {
    return Pair{cfma1(a.re, s, b.re), cfma1(a.im, s, b.im)};
}

// NL = a^2 e + 2 |a|^2 conj(e) with e = carrier z; with w = a e this is
// a (3 Re w - i Im w), 14 packed operations for two points.
__device__ __forceinline__ Pair nl_eval(const Pair& a, const Pair& cph, float2 z) {
    const float2 zx = dup2(z.x), zy = dup2(z.y), nzx = dup2(-z.x), nzy = dup2(-z.y);
    const float2 ex = fma2(cph.re, zx, mul2(cph.im, nzy));
    const float2 ney = fma2(cph.re, nzy, mul2(cph.im, nzx));
    const float2 nax = mul2(a.re, dup2(-1.f));
    const float2 wx = fma2(a.im, ney, mul2(a.re, ex));
    const float2 wy = fma2(nax, ney, mul2(a.im, ex));
    const float2 w3 = mul2(wx, dup2(3.f));
    return Pair{fma2(a.im, wy, mul2(a.re, w3)), fma2(nax, wy, mul2(a.im, w3))};
}

// K = -i hG (NL - i cs (NL[+1] - NL[-1]))
__device__ __forceinline__ Pair k_eval(const Pair& nlm, const Pair& nl0, const Pair& nlp, float hg, float cs) {
    const Pair d = pair_sub(nlp, nlm);
    return Pair{mul2(cfma1(d.re, -cs, nl0.im), dup2(hg)), mul2(cfma1(d.im, cs, nl0.re), dup2(-hg))};
}
// the same for one point
__device__ __forceinline__ float2 nl_one(float2 a, float2 cph, float2 z) {
    const Pair p = nl_eval(Pair{dup2(a.x), dup2(a.y)}, Pair{dup2(cph.x), dup2(cph.y)}, z);
    return make_float2(p.re.x, p.im.x);
}
__device__ __forceinline__ float2 k_one(float2 nlm, float2 nl0, float2 nlp, float hg, float cs) {
    const Pair p = k_eval(Pair{dup2(nlm.x), dup2(nlm.y)}, Pair{dup2(nl0.x), dup2(nl0.y)},
                          Pair{dup2(nlp.x), dup2(nlp.y)}, hg, cs);
    return make_float2(p.re.x, p.im.x);
}

// K of all H pairs of a thread from its drive and the neighbours' values L and R
template <int H>
__device__ __forceinline__ void k_all(const Pair (&nl)[H], float2 L, float2 R, float hg, float cs, Pair (&k)[H]) {
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const Pair m = j > 0 ? nl[j - 1]
                             : Pair{make_float2(L.x, nl[H - 1].re.x), make_float2(L.y, nl[H - 1].im.x)};
        const Pair p = j < H - 1 ? nl[j + 1]
                                 : Pair{make_float2(nl[0].re.y, R.x), make_float2(nl[0].im.y, R.y)};
        k[j] = k_eval(m, nl[j], p, hg, cs);
    }
}

__device__ __forceinline__ int time_index(int i, int n, int mode) {
    if (mode == TIME_SHIFTED) return (i > n / 2) ? i - n / 2 : i + n / 2;
    if (mode == TIME_NEE) return (i < n / 2) ? i : i - n;      // fftshift(t), NEE_CPU.m:12,53
    return i;
}

__device__ __forceinline__ float abc_factor(int i, int n, int mode) {
    if (mode == ABC_NONE) return 1.f;
    if (mode == ABC_NEE) {
        // NEE_CPU.m:114-121: 1 - sech^2(24 (1 - |2t| / range(t))) where
        // range(t) - |2t| < range(t) / 4, range(t) = (n - 1) dt, t = fftshift(t)
        const int it = (i < n / 2) ? i : i - n;
        const float r = 1.f - 2.f * fabsf((float)it) / (float)(n - 1);
        if (!(r < 0.25f)) return 1.f;
        const float th = tanhf(24.f * r);
        return th * th;
    }
    int gi1 = 6 * (n / 16), gi2 = 10 * (n / 16);
    if (!(i > gi1 && i < gi2)) return 1.f;
    if (mode == ABC_HARD) return 0.f;
    // 1 - sech^2(pos) evaluated as tanh^2(pos): no cancellation near the window edge
    float pos = (48.f * fabsf((float)i - 0.5f * (float)n)) / (float)n;
    float th = tanhf(pos);
    return th * th;
}

// Error class of one point: pct = scale |d| / (|e| + 1) against the percent
// thresholds (OPO_CUDA_BATCH_XTAL.cu:325-349; points with |e| == 0 skipped).
// Compared in squares so only |e| needs a square root.
__device__ __forceinline__ int classify(float scale, float2 d, float2 e, float maxE, float minE) {
    float e2 = e.x * e.x + e.y * e.y;
    int bits = 0;
    if (e2 > 0.f) {
        float den = sqrtf(e2) + 1.f;
        float lhs = scale * scale * (d.x * d.x + d.y * d.y);
        float hi = maxE * den, lo = minE * den;
        if (maxE <= 0.f || lhs >= hi * hi) bits = 1;
        else if (minE <= 0.f || lhs >= lo * lo) bits = 2;
    }
    if (!(isfinite(e.x) && isfinite(e.y))) bits |= 4;
    return bits;
}

// NEE_CPU.m:73-79 class: pct = scale |d| / (|e| + 1) over every point; bit 0
// when pct > maxErr (strict), bit 1 when pct >= minErr.
__device__ __forceinline__ int classify_nee(float scale, float2 d, float2 e, float maxE, float minE) {
    const float den = sqrtf(e.x * e.x + e.y * e.y) + 1.f;
    const float lhs = scale * scale * (d.x * d.x + d.y * d.y);
    const float hi = maxE * den, lo = minE * den;
    int bits = 0;
    if (lhs > hi * hi) bits |= 1;
    if (lhs >= lo * lo) bits |= 2;
    if (!(isfinite(e.x) && isfinite(e.y))) bits |= 4;
    return bits;
}

__device__ __forceinline__ float sqrt_fast(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// OR of the error classes of a thread's points, from E and d (pct = scale |d| / (|E| + 1)).
// The common case takes the largest q = |d|^2 / (|E| + 1)^2 by approximate square roots
// and reciprocals (relative error below 1e-6) and decides where q is more than 1e-5
// from both thresholds and below the upper one; everything else -- a point near or
// above a threshold, a non-finite, huge or vanishing field, non-positive bounds --
// goes through the exact classes, so every decision is theirs.  The exact class's IEEE
// square root costs more than the rest of a point's stage arithmetic.
struct Bounds {
    float qhi, qlo0, qlo1;
    Bounds() = default;
    __device__ Bounds(float scale, float hi, float lo) {
        const float is2 = 1.f / (scale * scale), l = lo > 0.f ? lo * lo * is2 : -1.f;
        qhi = hi > 0.f && lo > 0.f ? hi * hi * is2 * (1.f - 1e-5f) : -1.f;      // -1: always the exact classes
        qlo0 = l * (1.f - 1e-5f);
        qlo1 = l * (1.f + 1e-5f);
    }
};

template <int H, bool NEE>
__device__ __forceinline__ int classify_all(const Bounds& B, const PulseDev& P, float scale, const Pair (&d)[H],
                                            const Pair (&e)[H]) {
    float qmax = 0.f, emin = 3e38f;
    float2 sum = dup2(0.f);
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const float2 e2 = fma2(e[j].re, e[j].re, mul2(e[j].im, e[j].im));
        const float2 d2 = fma2(d[j].re, d[j].re, mul2(d[j].im, d[j].im));
        const float2 den = add2(make_float2(sqrt_fast(e2.x), sqrt_fast(e2.y)), dup2(1.f));
        const float2 r = make_float2(rcp_fast(den.x), rcp_fast(den.y));
        const float2 q = mul2(mul2(d2, r), r);
        qmax = fmaxf(qmax, fmaxf(q.x, q.y));
        emin = fminf(emin, fminf(e2.x, e2.y));
        sum = add2(sum, e2);
    }
    const float s = sum.x + sum.y;
    const bool low = qmax < B.qlo0, high = qmax > B.qlo1;
    if (s < 1e30f && qmax < B.qhi && (low || (high && (NEE || emin > 1e-30f)))) return high ? 2 : 0;
    int bits = 0;
    const float maxE = P.max_err, minE = P.min_err;
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const float2 d0 = make_float2(d[j].re.x, d[j].im.x), d1 = make_float2(d[j].re.y, d[j].im.y);
        const float2 e0 = make_float2(e[j].re.x, e[j].im.x), e1 = make_float2(e[j].re.y, e[j].im.y);
        bits |= NEE ? classify_nee(scale, d0, e0, maxE, minE) : classify(scale, d0, e0, maxE, minE);
        bits |= NEE ? classify_nee(scale, d1, e1, maxE, minE) : classify(scale, d1, e1, maxE, minE);
    }
    return bits;
}

// Phase rate beta (radians per step) as a 64-bit fixed-point fraction of a turn
__device__ __forceinline__ uint64_t phase_rate(float beta) {
    constexpr double kTwoPi = 6.283185307179586476925286766559, kTwoPiLo = 2.4492935982947064e-16;
    constexpr double kTurnScale = 18446744073709551616.0 / kTwoPi;   // 2^64 / (2 pi)
    const double b = (double)beta, n = rint(b * (1.0 / kTwoPi));
    double x = fma(-n, kTwoPiLo, fma(-n, kTwoPi, b)) * kTurnScale;
    if (x >= 9.2233720368547758e18) x -= 1.8446744073709552e19;
    if (x < -9.2233720368547758e18) x += 1.8446744073709552e19;
    return (uint64_t)(long long)llrint(x);
}

// D - 1 = alpha^s exp(-i th) - 1 for the phase increment d32 (units of 2^-32
// turn; converted to FP32, *dapplied receives the integer actually used) and
// log2 alpha l2 (-inf: alpha = 0).
__device__ __forceinline__ float2 dispersion_dm1(int d32, float l2, int s, int* dapplied) {
    if (l2 == -INFINITY) { *dapplied = d32; return make_float2(-1.f, 0.f); }
    float df = (float)d32;
    if (df >= 2147483648.f) df = 2147483520.f;
    *dapplied = __float2int_rn(df);
    float th = df * 1.4629180792671596e-09f;   // radians (2 pi 2^-32 per unit)
    float2 dm1;
    if (fabsf(th) < 0.25f) {
        // exp(-i th) - 1 by its Taylor series (no cancellation)
        float t2 = th * th;
        float cm1 = t2 * fmaf(t2, fmaf(t2, fmaf(t2, 2.48015873e-05f, -1.38888889e-03f), 4.16666667e-02f), -0.5f);
        float sn = th * fmaf(t2, fmaf(t2, fmaf(t2, -1.98412698e-04f, 8.33333333e-03f), -1.66666667e-01f), 1.f);
        dm1 = make_float2(cm1, -sn);
    } else {
        float s2, c2;
        sincospif(df * 0x1p-32f, &s2, &c2);   // sin, cos of th/2
        dm1 = make_float2(-2.f * s2 * s2, -2.f * s2 * c2);
    }
    if (l2 != 0.f) {
        float x = (float)s * l2;
        float as = exp2f(x);
        float am1 = expm1f(x * 0.69314718055994531f);
        dm1 = make_float2(fmaf(dm1.x, as, am1), dm1.y * as);
    }
    return dm1;
}

__device__ __forceinline__ float2 zphase(uint64_t tau_z4, float pos) {
    uint64_t p4 = (uint64_t)(uint32_t)(4.0f * pos);
    return turn_to_unit((uint64_t)0 - tau_z4 * p4);
}

// The z-phasors of up to three positions, one lane evaluating each
__device__ __forceinline__ void zphases(uint64_t tau_z4, int t, float p0, float p1, float p2, float2& z0, float2& z1,
                                        float2& z2) {
    const int l = t & 31;
    const float2 z = zphase(tau_z4, l == 0 ? p0 : (l == 1 ? p1 : p2));
    z0 = make_float2(__shfl_sync(0xffffffffu, z.x, 0), __shfl_sync(0xffffffffu, z.y, 0));
    z1 = make_float2(__shfl_sync(0xffffffffu, z.x, 1), __shfl_sync(0xffffffffu, z.y, 1));
    z2 = make_float2(__shfl_sync(0xffffffffu, z.x, 2), __shfl_sync(0xffffffffu, z.y, 2));
}

// ---------------------------------------------------------------------------
// shared-memory layout
// ---------------------------------------------------------------------------
// Cluster exchange: CTA c holds the n2 columns [c M/C, (c+1) M/C) of the C blocks.
// A thread takes PER consecutive columns whole, or, where there are fewer columns than
// threads (SPLIT), LANES consecutive lanes share a column: P values each, the C-point DFT as P-point DFTs in registers and a LANES-point one by
// shuffles.  (16 CTAs of 1024 points: two warps with 16 values a thread took 800 and
// 2190 cycles forward and inverse.)
template <int M, int C>
struct Xch {
    static constexpr int P = kPoints<M>, T = M / P;
    static constexpr int COLS = M / C;
    static constexpr bool SPLIT = COLS < T;
    static constexpr int LANES = SPLIT ? T / COLS : 1;
    static constexpr int PER = SPLIT ? 1 : COLS / T;
    static constexpr int NV = SPLIT ? P : PER * (C - 1);     // outer twiddles per thread
    // own parts of the exchange by plain stores and a block barrier (clusters of up to
    // 4, where they are a quarter or more of it), else through the cluster as the others
    static constexpr bool LOCAL = C <= 4;
    static constexpr int SEGT = COLS / P;                    // threads of a segment
};

// What a pass counts and only its records or the end of a trip need: kept by thread 0 in
// shared memory (the 4096-point kernels have 128 registers a thread, and spilled values
// wait on L2 beside 200 KB of shared memory).
struct RunState {
    double tally[4], prev_tally;
    unsigned long long grid_last[3];      // shared schedules: the grid's words after their last round
    int n_acc, n_rej, tot_att, tot_acc, tot_rej, steady, stop, slots, trips_done, status;
    // where registers are short: the next attempt's z-phasors and G sample, the classes' bounds
    float2 z[3];
    float g;
    Bounds bounds;
};

template <int M, int METHOD, int C>
struct Smem {
    static constexpr int P = kPoints<M>;
    static constexpr int T = M / P, NW = T / 32;
    using F = FftPlan<M, P>;
    using XC = Xch<M, C>;
    static constexpr size_t off_x = 0;                                               // stage output, FFT buffer
    static constexpr size_t off_g = off_x + sizeof(float2) * M;                      // clusters: gathered columns
    static constexpr size_t off_dm = off_g + (C > 1 ? sizeof(float2) * M : 0);       // per-mode D - 1
    static constexpr size_t off_tlo = off_dm + sizeof(float2) * M;                   // phase rates, low words
    static constexpr size_t off_abc = off_tlo + sizeof(uint32_t) * M;
    // absorber factors of the threads that have one (a quarter of them: the absorber spans
    // [6/16, 10/16] of the window in every variant), P each
    static constexpr size_t off_tw = off_abc + sizeof(float) * P * (T / 4 + 2);
    static constexpr size_t off_td = (off_tw + sizeof(float2) * F::TW + 15) & ~size_t(15);
    // exchange twiddles W_N^{n2 k1} and their d: [value][T]
    static constexpr size_t off_xtw = (off_td + sizeof(float) * F::TD + 15) & ~size_t(15);
    static constexpr size_t off_xtd = off_xtw + (C > 1 ? sizeof(float2) * XC::NV * T : 0);
    static constexpr size_t off_edge = (off_xtd + (C > 1 ? sizeof(float) * XC::NV * T : 0) + 15) & ~size_t(15);
    static constexpr size_t off_halo = off_edge + sizeof(float2) * 4 * NW;           // [parity][first, last][warp]
    // Heun: E and increment of the 4 halo points of every segment; RK23: the neighbours'
    // end values [parity][segment][left, right]
    // and, for a segment's two end threads, the field and the carrier of their halo points
    static constexpr size_t off_bar = off_halo + (C > 1 ? sizeof(float2) * (8 + 8) * C : 0);
    static constexpr size_t off_red = off_bar + sizeof(uint64_t) * 6;
    static constexpr size_t off_dred = off_red + sizeof(int) * (2 * NW + 2 * 16 + 8);   // warp and CTA flags, grid flags, waits that ran out
    static constexpr size_t off_run = ((off_dred + 15) & ~size_t(15)) + sizeof(double) * (NW * 4 + 2 * 16 * 4);
    static constexpr size_t bytes = off_run + sizeof(RunState);
    static_assert(bytes <= 232448 - 288, "shared memory of one CTA");
};

// ---------------------------------------------------------------------------
// cluster helpers
// ---------------------------------------------------------------------------
template <int C>
__device__ __forceinline__ void csync() {
    if constexpr (C > 1) cg::this_cluster().sync();
    else __syncthreads();
}

template <int C, typename Tp>
__device__ __forceinline__ Tp* remote(Tp* p, int rank) {
    if constexpr (C > 1) return cg::this_cluster().map_shared_rank(p, rank);
    else return p;
}

// 32-bit shared::cluster addressing: `mapa` turns a local shared address into the
// same offset in CTA `rank` of the cluster (half the registers of generic pointers)
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// ---------------------------------------------------------------------------
// Stores into a peer's shared memory that count their bytes on the peer's mbarrier
// (st.async): the receiver waits for exactly the bytes of one step of the exchange, with
// no fence and no cluster-wide barrier.  (32 KB all-to-all over 16 CTAs: 2370 cycles,
// against 3320 for plain remote stores and a cluster barrier; 4 KB over 8: 760, 1165.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void st_async(uint32_t addr, float2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, float2 v, float2 w, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr), "f"(v.x), "f"(v.y), "f"(w.x), "f"(w.y), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, int v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.s32 [%0], %1, [%2];" ::"r"(addr), "r"(v),
                 "r"(bar) : "memory");
}
__device__ __forceinline__ void bar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// the one arrival of a phase, with the bytes that complete it
__device__ __forceinline__ void bar_arm(uint32_t bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}

// Waits that run out.  dead[0]: a wait of this CTA ran out.  dead[kBars]: the cluster
// barriers of rejected steps and tallies so far; dead[kTold]: the number of the barrier at
// which a peer, whose wait ran out, leaves (0: none).
//  - A wait of steps B to E that ran out only sets dead[0]: the attempt goes on with what is
//    there (every branch depends on agreed flags alone), and the next attempt's flags, of
//    which dead[0] is one, end the pass in the whole cluster.
//  - The wait for the flags themselves (step A) is lost for all threads of a CTA or for none
//    (verdict_lost).  A CTA that loses it tells its peers the number of its last cluster
//    barrier; they are there or still run, so none has left.
//  - That barrier may pair with a peer's barrier of a rejected step or of the tallies.  The
//    word is visible behind it, in every CTA, so nobody sends anything any more.  (A word of
//    a later barrier may come in there too; it is another number.)
//  - A CTA that knows of a wait that ran out then stays for 2^20 cycles (peers' stores in
//    flight land in microseconds) and reports it.
//  - An mbarrier is armed again only after a phase of it that completed.
constexpr int kTold = 3, kBars = 4, kOut = 5, kVerdict = 6;
// whether the phase completed
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* dead, int limit) {
    while (!bar_try(bar, parity)) {
        if (--limit < 0 || dead[0]) {
            dead[0] = 1;
            return false;
        }
    }
    return true;
}
// the same, then thread 0 arms the next phase
__device__ __forceinline__ void bar_next(uint32_t bar, uint32_t parity, int bytes, volatile int* dead, int limit,
                                         int t) {
    if (bar_wait(bar, parity, dead, limit) && t == 0) bar_arm(bar, bytes);
}
// Where a thread's patience ran out: whether the phase is lost, the same for all T threads of
// the CTA without a barrier between them.  The threads count themselves in dead[kOut], and
// the last of all T looks once more and writes the verdict (1 complete, 2 lost).  A thread
// that finds the phase complete while the count is below T goes on, counted or not: whoever
// counts last looks later, and finds it complete too.
template <int T>
__device__ __noinline__ bool verdict_lost(uint32_t bar, uint32_t parity, volatile int* dead) {
    int verdict = 0;
    if (atomicAdd((int*)dead + kOut, 1) == T - 1) dead[kVerdict] = bar_try(bar, parity) ? 1 : 2;
    while (!verdict) {
        const bool done = bar_try(bar, parity);
        verdict = dead[kVerdict];
        if (!verdict && done && dead[kOut] < T) verdict = 1;
    }
    if (verdict == 2) dead[0] = 1;
    else if (atomicSub((int*)dead + kOut, 1) == 1) dead[kVerdict] = 0;      // none left: for the next phase
    return verdict == 2;
}
// The wait for the flags.  (A block-wide OR behind an ordinary wait took clusters 5 to 8 %:
// 4096 points on 8 CTAs 3.3 -> 3.5 us an attempt; the verdict's code inlined 2 %.)
template <int T>
__device__ __forceinline__ bool flags_lost(uint32_t bar, uint32_t parity, volatile int* dead, int limit) {
    do {
        if (bar_try(bar, parity)) return false;
    } while (--limit >= 0 && !dead[kTold]);
    return verdict_lost<T>(bar, parity, dead);
}
// before and behind a cluster barrier that may pair with a peer's last one
__device__ __forceinline__ void count_bar(int* dead, int t) {
    if (t == 0) ++dead[kBars];
}
__device__ __forceinline__ bool peer_gone(const volatile int* dead) {
    return dead[kTold] != 0 && dead[kTold] == dead[kBars];
}
// The two parts around the last cluster barrier.  Thread and rank are read again here: kept to
// the end of the pass they cost the 4096-point kernels registers that they do not have.
template <int C>
__device__ __forceinline__ int2 whoami() {
    int t, c = 0;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    if constexpr (C > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(c));
    return make_int2(t, c);
}
// before: the word to the peers, where a wait ran out; returns whether the barrier is to be
// left out, as the last one met a peer's last
template <int C>
__device__ __forceinline__ bool last_word(int* dead) {
    __syncthreads();
    if constexpr (C > 1) {
        if (dead[0] | dead[kTold]) {
            if (peer_gone(dead)) return true;
            const int2 me = whoami<C>();
            if (me.x < C && me.x != me.y) *cg::this_cluster().map_shared_rank(dead + kTold, me.x) = dead[kBars] + 1;
        }
    }
    return false;
}
// behind: if a wait of the cluster ran out, the field is NaN (the one sign that a caller without
// a status has) and the status says so
template <int M, int C, typename V>
__device__ __forceinline__ void end_lost(const volatile int* dead, V* out, optifax_pulse_stats* stats, const KernelCfg& cfg) {
    if (!(dead[0] | dead[kTold])) return;
    __syncthreads();                   // behind the stores of the field
    if (C > 1)
        for (const long long t0 = clock64(); clock64() - t0 < (1 << 20);) {}
    const int2 me = whoami<C>();
    V nan;
    nan.x = nan.y = __int_as_float(0x7fc00000);
#pragma unroll 1
    for (int i = me.x; i < M; i += blockDim.x) out[me.y * M + i] = nan;
    if (me.x == 0 && me.y == 0) {
        if (cfg.shared_sched) atomicOr(cfg.grid_sync + 3, 1ull);
        if (stats) {
            *stats = optifax_pulse_stats{};
            stats->status = OPTIFAX_PULSE_TIMEOUT;
        }
    }
}

// The neighbours' adjacent drive values: shuffles inside a warp, one shared-memory slot
// per warp edge where a segment is longer than a warp's points.  The ends of a segment
// wrap around (one CTA) or are replaced by the caller.
template <int M, int C>
__device__ __forceinline__ void exchange_edges(float2* edge, int& par, int t, float2 first, float2 last, float2& left,
                                               float2& right) {
    constexpr int NW = M / kPoints<M> / 32;
    const int w = t >> 5, lane = t & 31;
    left = make_float2(__shfl_up_sync(0xffffffffu, last.x, 1), __shfl_up_sync(0xffffffffu, last.y, 1));
    right = make_float2(__shfl_down_sync(0xffffffffu, first.x, 1), __shfl_down_sync(0xffffffffu, first.y, 1));
    if constexpr (Xch<M, C>::SEGT > 32) {
        float2* e = edge + par * 2 * NW;
        if (lane == 0) e[w] = first;
        if (lane == 31) e[NW + w] = last;
        __syncthreads();
        if (lane == 0) left = e[NW + (w > 0 ? w - 1 : NW - 1)];
        if (lane == 31) right = e[w < NW - 1 ? w + 1 : 0];
    }
    par ^= 1;
}

// N-point twiddle W_N^e, 0 <= e < N = C M, from the two tables: W_M^{(64/C)(e >> 6)}
// (quarter table, exact) times W_N^{e & 63}.  The product is rounded once; the inverse
// multiplies by its exact reciprocal conj(w)(1 + d), d = 1/|w|^2 - 1 formed from w
// itself, so forward + inverse carry no gain.
template <int M, int C>
__device__ __forceinline__ float2 twn_val(const Twiddle* quad, const Twiddle* low, int e) {
    static_assert(64 % C == 0, "cluster size must divide 64");
    const Twiddle a = quad_tw<M>(quad, (64 / C) * (e >> 6));
    const Twiddle b = low[e & 63];
    return cmul(make_float2(a.c, a.s), make_float2(b.c, b.s));
}

// Four-step split of the N = C M transform across a cluster through distributed shared
// memory.  Every value is pushed into the shared memory of the CTA that uses it next;
// each step has one mbarrier per CTA that counts the bytes the CTA gets in it:
//   A  the error flags and the halo points' E
//   B  exchange_fwd  C-point DFTs of the own columns (buffer g), twiddle -> the blocks' owners (x)
//   C  push_inverse  the last inverse pass's outputs -> the columns' owners (g)
//   D  exchange_inv  inverse twiddle and C-point DFTs, 1/N -> own points (x); the halo
//                    points' increments
// No buffer is written before its last read: what a CTA sends in a step carries what all
// of its threads read before (every thread adds to every peer's bytes of A, through the
// flags behind a block barrier, and of C; every reader of g to those of B).
// Store `v` (PER consecutive columns n2 of block k) into the FFT buffer of CTA k
template <int PER, bool LOCAL>
__device__ __forceinline__ void push_block(float2* bufx, uint32_t x, uint32_t bar, int k, int n2, const float2 (&v)[PER],
                                           int c) {
    const int s0 = swz(n2);
    if (LOCAL && k == c) {
#pragma unroll
        for (int u = 0; u < PER; ++u) bufx[s0 ^ u] = v[u];
        return;
    }
    const uint32_t dst = cluster_addr(x, k), db = dst + (bar - x);
    if constexpr (PER == 1) {
        st_async(dst + 8 * s0, v[0], db);
    } else {
#pragma unroll
        for (int u = 0; u < PER; u += 2) st_async(dst + 8 * (s0 ^ u), v[u], v[u + 1], db);
    }
}

__device__ __forceinline__ float2 shfl_xor2(float2 v, int m) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}
// LANES-point DFT across the lanes of a column (lane l ends with output bitrev(l)), and
// its exact reverse; one packed add or subtract per butterfly side.
template <int LANES, int NV>
__device__ __forceinline__ void lanes_fwd(float2 (&v)[NV], int l) {
#pragma unroll
    for (int hr = LANES / 2; hr >= 1; hr >>= 1) {
        const bool up = (l & hr) != 0;
        const bool turn = LANES == 4 && hr == 2 && (l & 1);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float2 o = shfl_xor2(v[i], hr);
            float2 d = up ? sub2(o, v[i]) : add2(v[i], o);
            if (up && turn) d = make_float2(d.y, -d.x);
            v[i] = d;
        }
    }
}
template <int LANES, int NV>
__device__ __forceinline__ void lanes_inv(float2 (&v)[NV], int l) {
#pragma unroll
    for (int hr = 1; hr <= LANES / 2; hr <<= 1) {
        const bool up = (l & hr) != 0;
        const bool turn = LANES == 4 && hr == 2 && (l & 1);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (up && turn) v[i] = make_float2(-v[i].y, v[i].x);
            const float2 o = shfl_xor2(v[i], hr);
            v[i] = up ? sub2(o, v[i]) : add2(v[i], o);
        }
    }
}

// Inner twiddles W_C^{j ka} of a lane's values (SPLIT), with their reciprocals' d: in
// registers, or, for two lanes of 8 values, the constants of the 16-point DFT by a select
// (at 4096 points per CTA 512 threads leave 128 registers, of which the table held 24:
// half of what that kernel spilled, and beside 220 KB of shared memory a spill is an L2
// access).
template <int M, int C>
struct Inner {
    static constexpr int P = kPoints<M>, LANES = Xch<M, C>::LANES;
    static constexpr bool SPLIT = Xch<M, C>::SPLIT, CONST = SPLIT && LANES == 2 && P == 8;
    float2 w[SPLIT && !CONST ? P : 1];
    float d[SPLIT && !CONST ? P : 1];
    __device__ __forceinline__ void fill(const Twiddle* quad, int t) {
        if constexpr (SPLIT && !CONST) {
#pragma unroll
            for (int r = 0; r < P; ++r) {
                const Twiddle a = quad_tw<M>(quad, ((t % LANES) * brev4(r, ilog2(P))) * (M / C) % M);
                w[r] = make_float2(a.c, a.s);
                d[r] = a.d;
            }
        }
    }
    // v times the twiddle of value r of lane l, and v over it
    __device__ __forceinline__ float2 mul(float2 v, int r, int l) const {
        if constexpr (CONST) {
            const float2 u = rot_fwd(v, brev4(r, 3));
            return l ? u : v;
        } else {
            return cmul(w[r], v);
        }
    }
    __device__ __forceinline__ float2 div(float2 v, int r, int l) const {
        if constexpr (CONST) {
            const float2 u = rot_inv(v, brev4(r, 3));
            return l ? u : v;
        } else {
            return mul_recip(v, w[r], d[r]);
        }
    }
};

// k1 of outer twiddle i of thread t (register i of the forward DFT)
template <int M, int C>
__device__ __forceinline__ int outer_k1(int i, int t) {
    using XC = Xch<M, C>;
    if constexpr (XC::SPLIT) return brev4(i, ilog2(XC::P)) + XC::P * brev4(t % XC::LANES, ilog2(XC::LANES));
    else return brev4(i % (C - 1) + 1, ilog2(C));
}

template <int M, int C>
__device__ __forceinline__ void exchange_fwd(const float2* g, float2* bufx, uint32_t x, uint32_t bar, const float2* xtw,
                                             const Inner<M, C>& in, int t, int c) {
    using XC = Xch<M, C>;
    if constexpr (XC::SPLIT) {
        constexpr int P = XC::P;
        const int l = t % XC::LANES, col = t / XC::LANES;
        float2 v[P];
#pragma unroll
        for (int i = 0; i < P; ++i) v[i] = g[swz((i * XC::LANES + l) * XC::COLS + col)];
        dftp<P>(v);
#pragma unroll
        for (int r = 1; r < P; ++r) v[r] = in.mul(v[r], r, l);
        lanes_fwd<XC::LANES, P>(v, l);
#pragma unroll
        for (int r = 0; r < P; ++r) {
            const float2 o[1] = {cmul(v[r], xtw[r * XC::T + t])};
            push_block<1, XC::LOCAL>(bufx, x, bar, outer_k1<M, C>(r, t), c * XC::COLS + col, o, c);
        }
    } else {
        float2 v[XC::PER][C];
        const int n2 = c * XC::COLS + t * XC::PER;
#pragma unroll
        for (int n1 = 0; n1 < C; ++n1) {
            const int s0 = swz(n1 * XC::COLS + t * XC::PER);
#pragma unroll
            for (int u = 0; u < XC::PER; ++u) v[u][n1] = g[s0 ^ u];
        }
#pragma unroll
        for (int u = 0; u < XC::PER; ++u) {
            dftp<C>(v[u]);
#pragma unroll
            for (int r = 1; r < C; ++r) v[u][r] = cmul(v[u][r], xtw[(u * (C - 1) + r - 1) * XC::T + t]);
        }
#pragma unroll
        for (int r = 0; r < C; ++r) {
            float2 o[XC::PER];
#pragma unroll
            for (int u = 0; u < XC::PER; ++u) o[u] = v[u][r];
            push_block<XC::PER, XC::LOCAL>(bufx, x, bar, brev4(r, ilog2(C)), n2, o, c);
        }
    }
}

// The segments next to segment `seg` of CTA c: their CTA, and their index there
template <int C>
__device__ __forceinline__ int seg_left(int seg, int c) { return c > 0 ? seg : (seg + C - 1) % C; }
template <int C>
__device__ __forceinline__ int seg_right(int seg, int c) { return c < C - 1 ? seg : (seg + 1) % C; }

// Increment of one of a segment's first or last two points for the neighbour's halo:
// halo[4 seg + 0..1] hold the points -2, -1 and halo[4 seg + 2..3] the points COLS,
// COLS + 1 of segment seg.
template <int M, int C>
__device__ __forceinline__ void push_halo(uint32_t halo, uint32_t bar, int seg, int col, float2 v, int c) {
    constexpr int COLS = Xch<M, C>::COLS;
    if (col >= 2 && col < COLS - 2) return;
    const bool first = col < 2;
    const uint32_t dst = cluster_addr(halo, first ? (c + C - 1) % C : (c + 1) % C);
    const int slot = first ? 4 * seg_left<C>(seg, c) + 2 + col : 4 * seg_right<C>(seg, c) + col - (COLS - 2);
    st_async(dst + 8 * slot, v, dst + (bar - halo));
}

template <int M, int C, bool HALO>
__device__ __forceinline__ void exchange_inv(const float2* g, float2* bufx, uint32_t halo, uint32_t bar, const float2* xtw,
                                             const float* xtd, const Inner<M, C>& in, int t, int c, float invN) {
    using XC = Xch<M, C>;
    if constexpr (XC::SPLIT) {
        constexpr int P = XC::P;
        const int l = t % XC::LANES, col = t / XC::LANES;
        float2 v[P];
#pragma unroll
        for (int r = 0; r < P; ++r) {
            v[r] = g[swz(outer_k1<M, C>(r, t) * XC::COLS + col)];
            v[r] = mul_recip(v[r], xtw[r * XC::T + t], xtd[r * XC::T + t]);
        }
        lanes_inv<XC::LANES, P>(v, l);
#pragma unroll
        for (int r = 1; r < P; ++r) v[r] = in.div(v[r], r, l);
        dftp_inv<P>(v);
        const bool ends = HALO && (col < 2 || col >= XC::COLS - 2);
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int n1 = i * XC::LANES + l;
            v[i] = mul2(v[i], dup2(invN));
            bufx[swz(n1 * XC::COLS + col)] = v[i];
            if (ends) push_halo<M, C>(halo, bar, n1, col, v[i], c);
        }
    } else {
        float2 v[XC::PER][C];
        const int col = t * XC::PER;
#pragma unroll
        for (int n1 = 0; n1 < C; ++n1) {
            const int s0 = swz(n1 * XC::COLS + col);
#pragma unroll
            for (int u = 0; u < XC::PER; ++u) v[u][n1] = g[s0 ^ u];
        }
#pragma unroll
        for (int u = 0; u < XC::PER; ++u) {
            float2 w[C];
            w[0] = v[u][0];
#pragma unroll
            for (int r = 1; r < C; ++r) {               // register r of the inverse DFT holds k1 = bitrev(r)
                const int i = (u * (C - 1) + r - 1) * XC::T + t;
                w[r] = mul_recip(v[u][brev4(r, ilog2(C))], xtw[i], xtd[i]);
            }
            dftp_inv<C>(w);
#pragma unroll
            for (int n1 = 0; n1 < C; ++n1) v[u][n1] = mul2(w[n1], dup2(invN));
        }
        const bool ends = HALO && (col < 2 || col + XC::PER > XC::COLS - 2);
#pragma unroll
        for (int n1 = 0; n1 < C; ++n1) {
            const int s0 = swz(n1 * XC::COLS + col);
#pragma unroll
            for (int u = 0; u < XC::PER; ++u) {
                bufx[s0 ^ u] = v[u][n1];
                if (ends) push_halo<M, C>(halo, bar, n1, col + u, v[u][n1], c);
            }
        }
    }
}

// The last inverse pass's outputs (points t + q M/P of this CTA's block) into the g
// buffers of their columns' owners.
template <int M, int C>
__device__ __forceinline__ void push_inverse(float2* bufg, uint32_t g, uint32_t bar, const float2 (&v)[kPoints<M>], int t,
                                             int c) {
    using XC = Xch<M, C>;
    constexpr int P = kPoints<M>;
    // with more CTAs than points a thread does not add to every peer's bytes, which then
    // say nothing about its reads of the FFT buffer
    if constexpr (C > P) __syncthreads();
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const int m = t + q * (M / P), r = m / XC::COLS, i = swz(c * XC::COLS + m % XC::COLS);
        if (XC::LOCAL && r == c) {
            bufg[i] = v[q];
        } else {
            const uint32_t dst = cluster_addr(g, r);
            st_async(dst + 8 * i, v[q], dst + (bar - g));
        }
    }
}

// OR of the error flags over the pulse: one slot per warp, then (clusters) one per CTA.
// Double buffered by attempt.  The barrier inside also publishes what the threads
// stored before it (stage output, pushed columns).
constexpr int kDead = 8;          // a bounded wait ran out: the same in every thread of the CTA

// The same over every pulse of a shared schedule (a cooperative launch).  One 64-bit word
// per attempt, three in turn, counts the clusters that have arrived and, per flag, those
// that raised it: one atomic add per cluster and one polling thread per CTA (a
// cooperative-groups grid barrier with a separate flag word took 5 us an attempt).  The
// words only grow: a round is the difference to the word's last total, so nothing is
// cleared between rounds, nothing but the word itself is communicated, and relaxed
// accesses do (a word is used again only once every CTA has read its last round).  Six
// pulses of 2048 points, us per attempt: 4.1 with release and acquire accesses and cleared
// words, 3.65 so; one pulse alone 3.35.
__device__ __forceinline__ int combine_grid(int f, int* slot, unsigned long long* last, int* dead, int attempt, int t,
                                            int c, const KernelCfg& cfg) {
    const int i = attempt % 3;
    unsigned long long* w = cfg.grid_sync + i;
    if (t == 0) {
        if (c == 0) {
            const unsigned long long v = 1ull + ((unsigned long long)(f & 1) << 16) +
                                         ((unsigned long long)((f >> 1) & 1) << 32) +
                                         ((unsigned long long)((f >> 2) & 1) << 48);
            asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
        }
        last += i;
        int limit = 16 * cfg.wait;         // a look takes 0.2 us or more
        unsigned long long v;
        for (;;) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
            v -= *last;
            if ((int)(v & 0xffffu) == cfg.clusters) break;
            if (--limit < 0) {
                *dead = 1;
                f |= kDead;
                break;
            }
        }
        *last += v;
        slot[attempt & 1] = ((v >> 16) & 0xffffu ? 1 : 0) | ((v >> 32) & 0xffffu ? 2 : 0) | ((v >> 48) ? 4 : 0) | (f & kDead);
    }
    __syncthreads();
    return slot[attempt & 1];
}

template <int NW, int C>
__device__ __forceinline__ int combine_flags(int bits, int* red, uint32_t bar, uint32_t parity, int bytes, int* dead,
                                             unsigned long long* last, int attempt, int t, int c, const KernelCfg& cfg) {
    const int par = attempt & 1;
    int* wf = red + par * NW;
    if (C > 1 && *(volatile int*)dead) bits |= kDead;
    const int w = __reduce_or_sync(0xffffffffu, bits);
    if ((t & 31) == 0) wf[t >> 5] = w;
    __syncthreads();
    int f = 0;
    if constexpr (NW >= 4) {
#pragma unroll
        for (int i = 0; i < NW; i += 4) {
            const int4 q = *reinterpret_cast<const int4*>(wf + i);
            f |= q.x | q.y | q.z | q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NW; ++i) f |= wf[i];
    }
    if constexpr (C > 1) {
        int* cl = red + 2 * NW + par * 16;
        if (t < C && t != c) {
            const uint32_t src = smem_u32(cl + c), dst = cluster_addr(src, t);
            st_async(dst, f, dst + (bar - src));
        }
        if (flags_lost<32 * NW>(bar, parity, dead, cfg.wait)) return kDead;
        if (t == 0) bar_arm(bar, bytes);
#pragma unroll
        for (int r = 0; r < C; ++r)
            if (r != c) f |= cl[r];
        if (f & kDead) {
            if (t == 0) *dead = 1;
            return kDead;
        }
    }
    if (cfg.shared_sched) f = combine_grid(f, red + 2 * NW + 2 * 16 + 1, last, dead, attempt, t, c, cfg);
    return f;
}

// ---------------------------------------------------------------------------
// FP64 sum of 4 per-thread values over the CTA and the cluster; every thread
// of every CTA returns the same totals (ranks summed in a fixed order).
// ---------------------------------------------------------------------------
template <int M, int C>
__device__ __forceinline__ void reduce_tallies(const float (&part)[4], double (&out)[4], double* dred,
                                               int t, int c, int parity) {
    constexpr int T = M / kPoints<M>, NW = T / 32;
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[i] = (double)part[i];
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    }
    if ((t & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) dred[(t >> 5) * 4 + i] = v[i];
    }
    __syncthreads();
    double* cl = dred + NW * 4 + parity * 16 * 4;
    if (t == 0) {
        double s[4] = {0, 0, 0, 0};
        for (int w = 0; w < NW; ++w)
            for (int i = 0; i < 4; ++i) s[i] += dred[w * 4 + i];
        for (int r = 0; r < C; ++r) {
            double* dst = remote<C>(cl, r) + c * 4;
            for (int i = 0; i < 4; ++i) dst[i] = s[i];
        }
    }
    csync<C>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double s = 0.0;
        for (int r = 0; r < C; ++r) s += cl[r * 4 + i];
        out[i] = s;
    }
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// One launch runs n_trips crystal passes of every pulse.  With a round-trip
// transfer (OPO mode, reference OpticalSim.run, OpticalSim.m:230-288) the last
// accepted step of each pass maps its spectrum X through the cavity,
// Y = X fb + pump, and the next pass starts from IFFT(Y): refraction into
// and out of the crystal, the intracavity optics, the output coupler, the
// delay and the pump injection are all per-mode products folded into fb and
// pump by the host.  Per-trip energy tallies sum tally_w |X|^2 in FP64.
template <int M, int C, int METHOD>
__global__ void __launch_bounds__(M / kPoints<M>, 1)
pass_kernel(const PulseDev* __restrict__ pulses, FftTables tabs, KernelCfg cfg) {
    constexpr int P = kPoints<M>, H = P / 2;
    constexpr int T = M / P;
    constexpr int N = M * C;
    constexpr int LOG2M = ilog2(M);
    constexpr bool nee = (METHOD == kHeunNee);   // NEE_CPU.m: k is 1-based, no chunk clamp
    constexpr bool heun = (METHOD != OPTIFAX_RK23);
    // clusters, Heun: the two points beyond each end of the CTA's block are carried
    // along by the end threads, so the stages need no exchange between CTAs
    constexpr bool HALO = heun && C > 1;
    using SM = Smem<M, METHOD, C>;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* bufX = reinterpret_cast<float2*>(smem + SM::off_x);
    float2* bufG = reinterpret_cast<float2*>(smem + SM::off_g);
    float2* dm_s = reinterpret_cast<float2*>(smem + SM::off_dm);
    uint32_t* tlo_s = reinterpret_cast<uint32_t*>(smem + SM::off_tlo);
    float* abc_s = reinterpret_cast<float*>(smem + SM::off_abc);
    float2* tw_s = reinterpret_cast<float2*>(smem + SM::off_tw);
    float* td_s = reinterpret_cast<float*>(smem + SM::off_td);
    float2* xtw_s = reinterpret_cast<float2*>(smem + SM::off_xtw);
    float* xtd_s = reinterpret_cast<float*>(smem + SM::off_xtd);
    float2* edge = reinterpret_cast<float2*>(smem + SM::off_edge);
    float2* halo_e = reinterpret_cast<float2*>(smem + SM::off_halo);      // E of every segment's halo points
    float2* halo_d = halo_e + 4 * C;                                      // their increments
    float2* ends = halo_e;                                                // RK23: [parity][segment][left, right]
    int* red = reinterpret_cast<int*>(smem + SM::off_red);
    int* dead = red + 2 * SM::NW + 2 * 16;
    double* dred = reinterpret_cast<double*>(smem + ((SM::off_dred + 15) & ~size_t(15)));
    RunState* run = reinterpret_cast<RunState*>(smem + SM::off_run);

    const int t = threadIdx.x;
    const int c = (C > 1) ? (int)cg::this_cluster().block_rank() : 0;
    const int p = blockIdx.x / C;
    // The descriptor is read all through the loop; a shared-memory copy keeps
    // those reads off the global path (and out of reach of aliasing with the
    // kernel's global stores).
    __shared__ PulseDev sP;
    if (t == 0) {
        sP = pulses[p];
        dead[0] = dead[kTold] = dead[kBars] = dead[kOut] = dead[kVerdict] = 0;
        *run = RunState{};
        run->bounds = Bounds(METHOD != OPTIFAX_RK23 ? 50.f : 200.f, sP.max_err, sP.min_err);
    }
    __syncthreads();
    const PulseDev& P_ = sP;

    // ---- prologue -------------------------------------------------------
    fft_tables<M, P>(tw_s, td_s, tabs.quad, t);
    if constexpr (C > 1) {
        using XC = Xch<M, C>;
#pragma unroll 1
        for (int i = 0; i < XC::NV; ++i) {
            const int n2 = c * XC::COLS + (XC::SPLIT ? t / XC::LANES : t * XC::PER + i / (C - 1));
            const float2 w = twn_val<M, C>(tabs.quad, tabs.low, n2 * outer_k1<M, C>(i, t));
            xtw_s[i * XC::T + t] = w;
            xtd_s[i * XC::T + t] = inv_norm2_m1(w);
        }
    }
    Inner<M, C> inner;
    if constexpr (C > 1) inner.fill(tabs.quad, t);
    // barriers of the exchange steps A to D, and of RK23's end values [parity]; bytes that
    // a CTA gets in each
    using XC_ = Xch<M, C>;
    constexpr int kAll = 8 * (XC_::LOCAL ? M - XC_::COLS : M);
    constexpr int kBytesA = 4 * (C - 1) + (HALO ? 32 * C : 0), kBytesD = 32 * C, kBytesE = 16 * C;
    const uint32_t bars = smem_u32(smem + SM::off_bar);
    const uint32_t bar_a = bars, bar_b = bars + 8, bar_c = bars + 16, bar_d = bars + 24, bar_e = bars + 32;
    if (C > 1 && t == 0) {
        for (int i = 0; i < 6; ++i) bar_init(bars + 8 * i);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_arm(bar_a, kBytesA);
        bar_arm(bar_b, kAll);
        bar_arm(bar_c, kAll);
        bar_arm(bar_d, kBytesD);
        bar_arm(bar_e, kBytesE);
        bar_arm(bar_e + 8, kBytesE);
    }
    uint32_t ph_x = 0, ph_e = 0;      // phase parities: B to D, end values (bit per parity); A: the attempt's
    // per-thread tables as vectors of four (or two) values: [j / 4][t][j % 4]
    auto at4 = [&](int j) { return ((j >> 2) * T + t) * 4 + (j & 3); };
    auto at2 = [&](int j) { return ((j >> 1) * T + t) * 2 + (j & 1); };
    auto carrier = [&](int i) { return turn_to_unit(P_.tau_theta * (uint64_t)time_index(i, N, cfg.time_mode)); };
    // this thread's points: i0 .. i0 + P-1; its place in a segment
    const int seg = t / XC_::SEGT, tin = t % XC_::SEGT;
    const int i0 = seg * M + c * XC_::COLS + P * tin;
    Pair a[H], cph[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const int i = i0 + j;
        const float2 c0 = carrier(i), c1 = carrier(i + H), e0 = P_.E_in[i], e1 = P_.E_in[i + H];
        cph[j] = Pair{make_float2(c0.x, c1.x), make_float2(c0.y, c1.y)};
        a[j] = Pair{make_float2(e0.x, e1.x), make_float2(e0.y, e1.y)};
    }
    float* abc = nullptr;                    // this thread's absorber factors, where it has any
    if (i0 + P > 6 * (N / 16) && i0 <= 10 * (N / 16) && cfg.abc_mode != ABC_NONE) {
        abc = abc_s + P * atomicAdd(&run->slots, 1);
#pragma unroll 1
        for (int j = 0; j < P; ++j) abc[j] = abc_factor(i0 + j, N, cfg.abc_mode);
    }
    // a segment's end threads: the adjacent (h1) and the outer (h2) point beyond its end
    const bool lend = C > 1 && tin == 0, rend = C > 1 && tin == XC_::SEGT - 1;
    // (field and carrier of both in shared memory: hs[0..1] and hs[2..3])
    float2* hs = halo_e + 8 * C + 4 * (2 * seg + (rend ? 1 : 0));
    if (HALO && (lend || rend)) {
        const int i1 = lend ? (i0 + N - 1) % N : (i0 + P) % N;
        const int i2 = lend ? (i0 + N - 2) % N : (i0 + P + 1) % N;
        hs[0] = P_.E_in[i1]; hs[1] = P_.E_in[i2];
        hs[2] = carrier(i1); hs[3] = carrier(i2);
    }
#pragma unroll 1
    for (int j = 0; j < P; ++j) {
        const int k = c + C * bitrev(P * t + j, LOG2M);
        const uint64_t tau = phase_rate(P_.beta[k]);
        tlo_s[at4(j)] = (uint32_t)tau;
    }
    if constexpr (C > 1) cg::this_cluster().sync(); else __syncthreads();

    // Values of the descriptor that every attempt uses: in registers, or read from shared
    // memory at each use where registers are short (4096 points per CTA)
    constexpr bool tight = T * 128 >= 65536;
    struct Hot { float h, cs, sel, S; int nchunks; const float* G; bool cavity; };
    auto load_hot = [&] { return Hot{P_.h, P_.c_shock, P_.sel, (float)P_.S, P_.nchunks, P_.G, P_.fb != nullptr}; };
    const Hot hot_ = load_hot();
    auto hot = [&]() -> Hot { if constexpr (tight) return load_hot(); else return hot_; };
    const Bounds bounds_ = tight ? Bounds{} : Bounds(heun ? 50.f : 200.f, P_.max_err, P_.min_err);
    auto bounds = [&]() -> Bounds { if constexpr (tight) return run->bounds; else return bounds_; };
    // what the caller asked for beyond the field, as one register (tested per attempt)
    constexpr int kForced = 1, kTrace = 2, kSteps = 4, kAp = 8;
    const int opts = (P_.forced && P_.n_forced > 0 ? kForced : 0) | (P_.trace ? kTrace : 0) |
                     (!nee && (P_.stepmods || P_.smt) ? kSteps : 0) | (P_.Ap ? kAp : 0);
    constexpr float invN = 1.0f / (float)N;
    const int guard = cfg.guard;
    const bool rec = (c == 0 && t == 0);
    const uint32_t x_addr = smem_u32(bufX), g_addr = smem_u32(bufG);

    float k = nee ? 1.f : 0.f, stepprev = 4.f, stepmod = 4.f;
    unsigned q = 0;                          // accumulated dispersion position (sum of stepmod)
    int s_cached = -1;                       // stepmod of the cached per-mode D - 1
    int par = 0, gatt = 0;                   // gatt: attempts of all trips

    // neighbours' drive values at the thread's ends; hv: the halo point's drive (end threads)
    auto edges = [&](const Pair (&nl)[H], float2 hv, float2& L, float2& R) {
        const float2 first = make_float2(nl[0].re.x, nl[0].im.x), last = make_float2(nl[H - 1].re.y, nl[H - 1].im.y);
        const int ep = par;
        if constexpr (C > 1 && !HALO) {
            // own end values to the neighbours; a slot is used again two exchanges later,
            // after its reader has sent its next values
            if (lend || rend) {
                const uint32_t src = smem_u32(ends + (ep * C + (lend ? seg_left<C>(seg, c) : seg_right<C>(seg, c))) * 2 +
                                              (lend ? 1 : 0));
                const uint32_t dst = cluster_addr(src, lend ? (c + C - 1) % C : (c + 1) % C);
                st_async(dst, lend ? first : last, dst + (bar_e + 8 * ep - src));
            }
        }
        exchange_edges<M, C>(edge, par, t, first, last, L, R);
        if constexpr (HALO) {
            if (lend) L = hv;
            if (rend) R = hv;
        } else if constexpr (C > 1) {
            if (lend || rend) {
                const uint32_t b = bar_e + 8 * ep;
                bar_next(b, (ph_e >> ep) & 1, kBytesE, dead, cfg.wait, t);
                (lend ? L : R) = ends[(ep * C + seg) * 2 + (lend ? 0 : 1)];
            }
            ph_e ^= 1u << ep;
        }
    };

    // z-phasors of an attempt's stages and its G sample, made ahead (before the
    // transforms of the previous step; ready: valid for the next attempt).  Where registers
    // are short warp 0 makes them, and they wait in shared memory.
    bool ready = false;                      // (where they are short; else keyed by position and step)
    float zk = -1.f, zs = -1.f, gval = 0.f;
    float2 z0 = make_float2(0.f, 0.f), z1 = z0, z2 = z0;
    auto phasors = [&](float kp, float sm) {
        if constexpr (heun) zphases(P_.tau_z4, t, kp, kp + sm, 0.f, z0, z1, z2);
        else zphases(P_.tau_z4, t, kp + 0.5f * sm, kp + 0.75f * sm, kp + sm, z0, z1, z2);
        gval = hot().G[(int)kp];
    };
    auto prepare = [&](float kp, float sm) {
        if constexpr (tight) {
            ready = true;
            if (t < 32) {
                phasors(kp, sm);
                if (t == 0) { run->z[0] = z0; run->z[1] = z1; run->z[2] = z2; run->g = gval; }
            }
        } else {
            phasors(kp, sm);
            zk = kp; zs = sm;
        }
    };

    Pair k1r[H];      // RK23: K1 (first stage, FSAL) between attempts
    do {
        k = nee ? 1.f : 0.f; stepprev = 4.f; stepmod = 4.f; q = 0;
        int trip_status = 0;
        int limit = gatt + cfg.max_attempts_mul * (P_.S + 16) + 64;     // of this trip's attempts
        if constexpr (!heun) {
            // initial K1 at k = 0 with stepmod = 4 (OPO_CUDA_ODE23.cu:432-438)
            const float hg = (stepmod * hot().h) * hot().G[0], cs = hot().cs;
            const float2 z = zphase(P_.tau_z4, 0.f);
            Pair nl[H];
#pragma unroll
            for (int j = 0; j < H; ++j) nl[j] = nl_eval(a[j], cph[j], z);
            float2 L, R;
            edges(nl, make_float2(0.f, 0.f), L, R);
            k_all<H>(nl, L, R, hg, cs, k1r);
        }

        // whether the pass goes on at position kk of a chunk that ends at ce
        auto more = [&](float kk, float ce) {
            const float Sf = hot().S;
            return kk < ce && (nee ? kk <= Sf : (!guard || kk < Sf));
        };
        for (int chunk = 0; chunk < hot().nchunks; ++chunk) {
            if (!nee) stepmod = stepprev;
            const float cend = (float)(chunk + 1) * hot().sel;
            while (more(k, cend)) {
                if (gatt >= limit) {
                    if (t == 0) run->status |= OPTIFAX_PULSE_ATTEMPT_LIMIT;
                    goto done;
                }
                const int krec = (int)k;
                // z of the first stage in steps and index of G (G33(k) is 1-based in NEE_CPU.m)
                const float kpos = nee ? k - 1.f : k;
                bool accepted = false;
                if constexpr (tight) {
                    if (ready) {
                        z0 = run->z[0]; z1 = run->z[1]; gval = run->g;
                        if constexpr (!heun) z2 = run->z[2];
                    } else {
                        phasors(kpos, stepmod);
                    }
                    ready = false;
                } else if (kpos != zk || stepmod != zs) {
                    prepare(kpos, stepmod);
                }
                const float hg = (stepmod * hot().h) * gval, cs = hot().cs;
                Pair ev[H];                                    // E, then E behind the absorber
                Pair dv[H];                                    // its error difference
                Pair k4[H];                                    // RK23: FSAL candidate
                if constexpr (heun) {
                    // ---- stage 1: K1 = f(A0) at z = k ----
                    Pair nl[H], k1[H], k2[H];
                    float2 L, R, zu = make_float2(0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < H; ++j) nl[j] = nl_eval(a[j], cph[j], z0);
                    float2 hn = make_float2(0.f, 0.f);
                    if (HALO && (lend || rend)) {
                        // drive and A1 of the adjacent halo point
                        const float2 h1 = hs[0], hc1 = hs[2];
                        const float2 n1 = nl_one(h1, hc1, z0), n2 = nl_one(hs[1], hs[3], z0);
                        const float2 in = lend ? make_float2(nl[0].re.x, nl[0].im.x)
                                               : make_float2(nl[H - 1].re.y, nl[H - 1].im.y);
                        const float2 kh = lend ? k_one(n2, n1, in, hg, cs) : k_one(in, n1, n2, hg, cs);
                        hn = n1;
                        zu = nl_one(cadd(h1, kh), hc1, z1);
                    }
                    edges(nl, hn, L, R);
                    k_all<H>(nl, L, R, hg, cs, k1);
                    // ---- stage 2: K2 = f(A0 + K1) at z = k + stepmod ----
#pragma unroll
                    for (int j = 0; j < H; ++j) nl[j] = nl_eval(pair_add(a[j], k1[j]), cph[j], z1);
                    edges(nl, zu, L, R);
                    k_all<H>(nl, L, R, hg, cs, k2);
                    // E = A0 + (K2/2 + K1/2) (MEX) or (A0 + K1/2) + K2/2 (NEE_CPU.m:75)
#pragma unroll
                    for (int j = 0; j < H; ++j) {
                        ev[j] = nee ? pair_fma(k2[j], 0.5f, pair_fma(k1[j], 0.5f, a[j]))
                                    : pair_fma(pair_add(k2[j], k1[j]), 0.5f, a[j]);
                        dv[j] = pair_sub(k2[j], k1[j]);                        // = 2 (E - A1)
                    }
                } else {
                    // ---- RK23: K2 at k + s/2, K3 at k + 3s/4, K4 at k + s (FSAL) ----
                    Pair nl[H], k2[H], pp[H];
                    float2 L, R;
#pragma unroll
                    for (int j = 0; j < H; ++j) nl[j] = nl_eval(pair_fma(k1r[j], 0.5f, a[j]), cph[j], z0);
                    edges(nl, make_float2(0.f, 0.f), L, R);
                    k_all<H>(nl, L, R, hg, cs, k2);
#pragma unroll
                    for (int j = 0; j < H; ++j) nl[j] = nl_eval(pair_fma(k2[j], 0.75f, a[j]), cph[j], z1);
                    edges(nl, make_float2(0.f, 0.f), L, R);
                    k_all<H>(nl, L, R, hg, cs, pp);
#pragma unroll
                    for (int j = 0; j < H; ++j) {
                        const Pair k3 = pp[j];
                        const float2 b1 = fma2(k2[j].re, dup2(1.f / 3.f), mul2(k3.re, dup2(4.f / 9.f)));
                        const float2 b2 = fma2(k2[j].im, dup2(1.f / 3.f), mul2(k3.im, dup2(4.f / 9.f)));
                        ev[j] = pair_fma(k1r[j], 2.f / 9.f, pair_add(a[j], Pair{b1, b2}));
                        // E - A1 without K4: (4/9-1/3) K3 + (1/3-1/4) K2 + (2/9-7/24) K1
                        const float2 c1 = fma2(k2[j].re, dup2(1.f / 12.f), mul2(k3.re, dup2(1.f / 9.f)));
                        const float2 c2 = fma2(k2[j].im, dup2(1.f / 12.f), mul2(k3.im, dup2(1.f / 9.f)));
                        pp[j] = pair_fma(k1r[j], -5.f / 72.f, Pair{c1, c2});
                    }
#pragma unroll
                    for (int j = 0; j < H; ++j) nl[j] = nl_eval(ev[j], cph[j], z2);
                    edges(nl, make_float2(0.f, 0.f), L, R);
                    k_all<H>(nl, L, R, hg, cs, k4);
#pragma unroll
                    for (int j = 0; j < H; ++j) dv[j] = pair_fma(k4[j], -1.f / 8.f, pp[j]);   // = E - A1
                }
                const int bits = classify_all<H, nee>(bounds(), P_, heun ? 50.f : 200.f, dv, ev);
                // E behind the absorber: into the FFT buffer, or the columns' buffer
                {
                    float2 o[P];
                    if (abc) {
#pragma unroll
                        for (int j = 0; j < H; ++j) {
                            const float2 f = make_float2(abc[j], abc[j + H]);
                            ev[j] = Pair{mul2(ev[j].re, f), mul2(ev[j].im, f)};
                        }
                    }
#pragma unroll
                    for (int j = 0; j < H; ++j) {
                        o[j] = make_float2(ev[j].re.x, ev[j].im.x);
                        o[j + H] = make_float2(ev[j].re.y, ev[j].im.y);
                    }
                    store_own<P>(C > 1 ? bufG : bufX, t, o);
                    if (HALO && (lend || rend)) {  // E of the end points: the neighbours' halos
                        const uint32_t src = smem_u32(halo_e + 4 * (lend ? seg_left<C>(seg, c) : seg_right<C>(seg, c)));
                        const uint32_t dst = cluster_addr(src, lend ? (c + C - 1) % C : (c + 1) % C);
                        const uint32_t db = dst + (bar_a - src);
                        if (lend) st_async(dst + 16, o[0], o[1], db);
                        else st_async(dst, o[P - 2], o[P - 1], db);
                    }
                }

                int fl = combine_flags<T / 32, C>(bits, red, bar_a, gatt & 1, kBytesA, dead, run->grid_last, gatt, t,
                                                  c, cfg);
                if (fl & kDead) goto done;
                if ((opts & kForced) && gatt < P_.n_forced) fl = (P_.forced[gatt] & 3) | (fl & 4);
                if (fl & 4) trip_status |= OPTIFAX_PULSE_NAN;

                if ((fl & 1) && stepmod > 1.f && (nee || (k - stepmod) > 0.f)) {
                    // ---- reject: A0 unchanged; MEX: k moves back by one in net (the loop
                    // adds the new stepmod); NEE: k stays (NEE_CPU.m:68-70)
                    if ((opts & kTrace) && rec && gatt < P_.trace_cap) {
                        P_.trace[3 * gatt] = krec; P_.trace[3 * gatt + 1] = (int)stepmod;
                        P_.trace[3 * gatt + 2] = fl & 7;
                    }
                    if (t == 0) ++run->n_rej;
                    if (!nee) k = k - stepmod;
                    stepmod = stepmod - 1.f;
                    stepprev = stepmod;
                    if constexpr (!heun) {
                        // K1 recomputed at z = k + stepmod with G[k] (OPO_CUDA_ODE23.cu:484-487)
                        const float hg1 = (stepmod * hot().h) * hot().G[(int)k];
                        const float2 z = zphase(P_.tau_z4, k + stepmod);
                        Pair nl[H];
                        float2 L, R;
#pragma unroll
                        for (int j = 0; j < H; ++j) nl[j] = nl_eval(a[j], cph[j], z);
                        edges(nl, make_float2(0.f, 0.f), L, R);
                        k_all<H>(nl, L, R, hg1, cs, k1r);
                    }
                    // the next attempt's flags and halos must not overtake this one's
                    if constexpr (C > 1) {
                        count_bar(dead, t);
                        cg::this_cluster().sync();
                        if (peer_gone(dead)) limit = 0;
                    }
                } else {
                    // ---- accept ----
                    if ((opts & kTrace) && rec && gatt < P_.trace_cap) {
                        P_.trace[3 * gatt] = krec; P_.trace[3 * gatt + 1] = (int)stepmod;
                        P_.trace[3 * gatt + 2] = (fl & 7) | 8;
                    }
                    if (t == 0) ++run->n_acc;
                    accepted = true;
                    const int s_used = (int)stepmod;
                    if ((opts & kSteps) && rec && krec < P_.stepmods_limit && krec < P_.S) {
                        if (P_.stepmods) P_.stepmods[krec] = (float)s_used;
                        if (P_.smt) P_.smt[(size_t)run->trips_done * P_.S + krec] = (float)s_used;
                    }
                    // step control (OPO_CUDA_BATCH_XTAL.cu:487-506; ODE23 :519-538 doubles;
                    // NEE_CPU.m:77-83: grow below minErr, clamp only at the crystal end)
                    if (nee) {
                        if (!(fl & 2)) stepmod = stepmod + 1.f;
                        const float Sf = hot().S;
                        if (k < Sf && k + stepmod > Sf) stepmod = Sf - k;
                    } else if (k + stepmod >= cend && k < cend - 1.f) {
                        float stepend = (cend - k) - 1.f;
                        stepprev = stepmod;
                        stepmod = stepend;
                    } else {
                        if constexpr (heun) {
                            if (!(fl & 2) && !(fl & 1) && (k + stepmod + 1.f) < cend - 1.f) stepmod = stepmod + 1.f;
                        } else {
                            if (!(fl & 2) && !(fl & 1) && (k + stepmod + stepmod) < cend - 1.f) stepmod = stepmod * 2.f;
                        }
                        stepprev = stepmod;
                    }
                    const float knext = k + stepmod;
                    const bool last_in_chunk = !more(knext, cend);
                    const bool pass_ends = !more(knext, (float)hot().nchunks * hot().sel);
                    const bool cav = pass_ends && hot().cavity;
                    const unsigned qn = q + (unsigned)s_used;

                    // ---- linear sub-step ----
                    // Incremental form: A_new = E + IFFT((D - 1) FFT(E)) / N with
                    // D = alpha^s exp(-i beta s): transform rounding then scales with
                    // |D - 1| instead of |E|.  At the end of an OPO pass the full
                    // spectrum goes through the cavity instead: A_new = IFFT(D FFT(E) fb + pump) / N.
                    if constexpr (C > 1) {
                        if (HALO && (lend || rend)) {
                            hs[0] = halo_e[4 * seg + (lend ? 1 : 2)];
                            hs[1] = halo_e[4 * seg + (lend ? 0 : 3)];
                        }
                        exchange_fwd<M, C>(bufG, bufX, x_addr, bar_b, xtw_s, inner, t, c);
                    }
                    // refresh the per-mode D - 1 when the step size changed (a compact loop:
                    // kept out of the unrolled mode loop below), for the exact fixed-point
                    // increment beta s: the FP32 rounding of its angle is applied as a
                    // first-order rotation, D e^{-i eps} - 1 ~ (D - 1) - i eps D
                    constexpr float kUnit = 1.4629180792671596e-09f;     // 2 pi 2^-32
                    if (s_used != s_cached) {
#pragma unroll 1
                        for (int j = 0; j < P; ++j) {
                            const int kk = c + C * bitrev(P * t + j, LOG2M);
                            const uint64_t tau = phase_rate(P_.beta[kk]);
                            const uint64_t inc = tau * (uint64_t)(unsigned)s_used;
                            const int d32 = (int)((long long)inc >> 32);
                            int dc;
                            const float l2 = log2f(P_.alpha[kk]);
                            const float2 m = dispersion_dm1(d32, l2, s_used, &dc);
                            const float e = (float)(int)((unsigned)d32 - (unsigned)dc) * kUnit;
                            dm_s[at2(j)] = make_float2(fmaf(e, m.y, m.x), fmaf(-e, 1.f + m.x, m.y));
                        }
                        s_cached = s_used;
                    }
                    if (!pass_ends) {
                        const float kn = nee ? knext - 1.f : knext;
                        prepare(kn, (!nee && last_in_chunk) ? stepprev : stepmod);
                    }
                    if constexpr (C > 1) {
                        if constexpr (XC_::LOCAL) __syncthreads();
                        bar_next(bar_b, ph_x, kAll, dead, cfg.wait, t);
                    }
                    float2 v[P];
                    fftp_forward<M, P>(bufX, tw_s, t, v);
                    float2* apc = (last_in_chunk && (opts & kAp)) ? P_.Ap + (size_t)chunk * N : nullptr;
                    float part[4] = {0.f, 0.f, 0.f, 0.f};
                    // the trip's crystal output goes to the cavity scratch; the cavity
                    // work (tallies, ESD sums, history, transfer) runs after the loop
                    float2* const xsp = cav ? P_.xs : nullptr;
                    uint32_t lo_[P];
                    float2 dm_[P];
#pragma unroll
                    for (int j = 0; j < P; j += 4) {
                        const uint4 w = *reinterpret_cast<const uint4*>(tlo_s + at4(j));
                        lo_[j] = w.x; lo_[j + 1] = w.y; lo_[j + 2] = w.z; lo_[j + 3] = w.w;
                    }
#pragma unroll
                    for (int j = 0; j < P; j += 2) {
                        const float4 w = *reinterpret_cast<const float4*>(dm_s + at2(j));
                        dm_[j] = make_float2(w.x, w.y);
                        dm_[j + 1] = make_float2(w.z, w.w);
                    }
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        // The step's phase is the difference of the two positions' exact
                        // fixed-point phases in units of 2^-32 turn: the cached increment's
                        // high word plus the carry of the low words' sum, tau qn = tau q + tau s.
                        const float e = (lo_[j] * qn < lo_[j] * (unsigned)s_used) ? kUnit : 0.f;
                        const float2 dm1 = make_float2(fmaf(e, dm_[j].y, dm_[j].x), fmaf(-e, 1.f + dm_[j].x, dm_[j].y));
                        const float2 eh = v[j];
                        if (apc || cav) {
                            const int kk = c + C * bitrev(P * t + j, LOG2M);
                            const float2 o = cadd(eh, cmul(eh, dm1));
                            if (apc) apc[kk] = o;
                            if (cav) xsp[kk] = o;
                        }
                        v[j] = cmul(eh, dm1);
                    }
                    if (cav) {
                        // once per round trip, outside the unrolled mode loop (code size):
                        // energy tallies, ESD sums and history of the crystal output X,
                        // then Y = X fb + pump; every mode has one owner thread, which
                        // reads back only what it wrote
#pragma unroll 1
                        for (int j = 0; j < P; ++j) {
                            const int kk = c + C * bitrev(P * t + j, LOG2M);
                            const float2 X = xsp[kk];
                            const float x2 = X.x * X.x + X.y * X.y;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (i < P_.n_tally) part[i] = fmaf(P_.tally_w[(size_t)i * N + kk], x2, part[i]);
#pragma unroll 1
                            for (int i = 0; i < P_.n_esd; ++i)
                                P_.esd[(size_t)i * N + kk] += P_.esd_w[(size_t)i * N + kk] * x2;
                            if (P_.hist) P_.hist[(size_t)run->trips_done * N + kk] = X;
                            xsp[kk] = cadd(cmul(X, P_.fb[kk]), P_.pump[kk]);
                        }
#pragma unroll
                        for (int j = 0; j < P; ++j) v[j] = xsp[c + C * bitrev(P * t + j, LOG2M)];
                    }
                    fftp_inverse<M, P>(bufX, tw_s, td_s, t, v);
                    if constexpr (C > 1) {
                        push_inverse<M, C>(bufG, g_addr, bar_c, v, t, c);
                        if constexpr (XC_::LOCAL) __syncthreads();
                        bar_next(bar_c, ph_x, kAll, dead, cfg.wait, t);
                        exchange_inv<M, C, HALO>(bufG, bufX, smem_u32(halo_d), bar_d, xtw_s, xtd_s, inner, t, c, invN);
                        __syncthreads();
                        if (HALO && (lend || rend)) {
                            bar_next(bar_d, ph_x, kBytesD, dead, cfg.wait, t);
                            const float2 d1 = halo_d[4 * seg + (lend ? 1 : 2)];
                            const float2 d2 = halo_d[4 * seg + (lend ? 0 : 3)];
                            hs[0] = cav ? d1 : cadd(hs[0], d1);
                            hs[1] = cav ? d2 : cadd(hs[1], d2);
                        }
                        ph_x ^= 1;
                    } else {
                        const int s0 = swz(t);
#pragma unroll
                        for (int i = 0; i < P; ++i) bufX[swz_at(s0, i * (M / P))] = v[i];
                        __syncthreads();
                    }
                    load_own<P>(bufX, t, v);
#pragma unroll
                    for (int j = 0; j < H; ++j) {
                        const Pair d{make_float2(v[j].x, v[j + H].x), make_float2(v[j].y, v[j + H].y)};
                        if constexpr (C > 1) a[j] = cav ? d : pair_add(ev[j], d);
                        else a[j] = cav ? Pair{mul2(d.re, dup2(invN)), mul2(d.im, dup2(invN))} : pair_fma(d, invN, ev[j]);
                        if constexpr (!heun) k1r[j] = k4[j];
                    }
                    if (cav) {
                        double tally[4];
                        count_bar(dead, t);
                        reduce_tallies<M, C>(part, tally, dred, t, c, run->trips_done & 1);
                        if (t == 0)
                            for (int i = 0; i < 4; ++i) run->tally[i] = tally[i];
                    }
                    q = qn;
                }
                ++gatt;
                if (!nee || accepted) k = k + stepmod;
            }
        }
        if (t == 0) {
            const int trip = run->trips_done, attempts = gatt - run->tot_att;
            run->status |= trip_status;
            if (rec && P_.fb && P_.trips) {
                optifax_trip_record tr;
                tr.attempts = attempts; tr.accepted = run->n_acc; tr.rejected = run->n_rej; tr.status = trip_status;
                for (int i = 0; i < 4; ++i) tr.tally[i] = run->tally[i];
                P_.trips[trip] = tr;
            }
            run->tot_att = gatt; run->tot_acc += run->n_acc; run->tot_rej += run->n_rej;
            run->n_acc = run->n_rej = 0;
            // steady state of a cavity: the totals are the same in every CTA of the cluster
            const double cur = run->tally[P_.steady_tally & 3];
            const bool flat = trip > 0 && cur != 0.0 &&
                              fabs(cur - run->prev_tally) <= (double)P_.steady_tol * fabs(cur);
            run->steady = flat ? run->steady + 1 : 0;
            run->prev_tally = cur;
            run->stop = trip + 1 >= P_.n_trips || (P_.fb && P_.steady_trips > 0 && run->steady >= P_.steady_trips) ||
                        (C > 1 && peer_gone(dead));
            run->trips_done = trip + 1;
            for (int i = 0; i < 4; ++i) run->tally[i] = 0.0;
        }
        __syncthreads();
    } while (!run->stop);
done:
    const bool gone = last_word<C>(dead);
#pragma unroll
    for (int j = 0; j < H; ++j) {
        P_.A_out[i0 + j] = make_float2(a[j].re.x, a[j].im.x);
        P_.A_out[i0 + j + H] = make_float2(a[j].re.y, a[j].im.y);
    }
    if (rec && P_.stats) {
        optifax_pulse_stats st;
        st.attempts = run->tot_att; st.accepted = run->tot_acc; st.rejected = run->tot_rej; st.status = run->status;
        st.z_steps = (long long)q; st.k_final = k; st.stepmod_final = stepmod; st.n_chunks = P_.nchunks;
        st.reserved[0] = run->trips_done; st.reserved[1] = st.reserved[2] = 0;
        *P_.stats = st;
    }
    if constexpr (C > 1) {
        if (!gone) cg::this_cluster().sync();        // no CTA leaves while a peer may still read its memory
    }
    end_lost<M, C>(dead, P_.A_out, P_.stats, cfg);
}

}  // namespace ofx
