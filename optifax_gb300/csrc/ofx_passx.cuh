// ofx_passx.cuh -- the persistent crystal-pass kernel with a wide field state.
//
// passx_kernel<R, M, C, NEE> runs the same Heun schedule as pass_kernel
// (ofx_pass.cuh; reference OPO_CUDA_BATCH_XTAL.cu:373-525 and its variants,
// NEE_CPU.m:1-122 with NEE) with every field value, stage sum and transform in
// the arithmetic type R:
//   R = double  the plain FP64 solver: the FP64 comparator of the FP32
//               propagator, computed as the FP64 oracle computes it;
//   R = ff      float-float (ofx_num.cuh), ~48-bit significands from FP32
//               operations, for high-gain passes in which FP32 rounding of the
//               field, amplified by the parametric gain, dominates the result.
// Layout, transforms and cluster exchange are pass_kernel's, in R: a cluster of C CTAs
// holds one pulse of N = C M points for the whole pass, each CTA its columns of every
// block, P consecutive points per thread (field A0 in registers), two-point halos at the
// segments' ends, exchanges pushed into the next user's shared memory and counted on its
// mbarriers.  Phases (carrier w0 t_i and z-carrier bdiffw0 z) are exact 64-bit
// fixed-point turns evaluated by FP64 sincospi; the dispersion factor and the absorber
// are FP64 (then rounded to R), as in the FP64 oracle.  The FP64 kernel is bound by
// GB300's FP64 pipe, the float-float kernel by issue and the cluster's latency.
#pragma once
#include <cooperative_groups.h>
#include <cstring>
#include <type_traits>
#include "ofx_num.cuh"
#include "ofx_pass.cuh"

namespace ofx {

// Per-pulse descriptor of the wide-state pass (device pointers).
struct PulseX {
    const double2* E_in;     // N complex doubles, fftshifted time
    double2* A_out;
    const double* alpha;     // N, FFT order
    const double* beta;      // N, FFT order
    const double* G;         // S
    int* trace;              // 3 ints per attempt (k, stepmod, flags | 8 accepted), or null
    optifax_pulse_stats* stats;
    void* ztab;              // scratch: zcap z-carrier phasors exp(-i bdiffw0 h p), p = 0..zcap-1, in R
    int zcap;
    uint64_t tau_theta;      // w0 dt in turns
    uint64_t tau_z;          // bdiffw0 h in turns (per z-sample)
    double w0, h, dt, max_err, min_err, sel, c_shock;
    int N, S, nchunks, trace_cap;
};

// W_N^e (N = C M) for e in [0, N), in R; the local transforms use W_M^e = W_N^{C e}.
template <typename R>
struct XTables { const typename Num<R>::cplx* wn; };

// exp(2 pi i u / 2^64) in FP64: the turn as a signed fraction in half-turns
__device__ __forceinline__ double2 turn_unit_d(uint64_t u) {
    const double x = (double)(long long)u * 0x1p-63;
    double s, c;
    sincospi(x, &s, &c);
    return make_double2(c, s);
}

// ---------------------------------------------------------------------------
// Shape of one kernel: P points per thread, exchange columns, transform passes.
// ---------------------------------------------------------------------------
template <int M, int C>
struct ShapeX {
    static constexpr int P = M >= 4096 ? 16 : (M >= 2048 ? 8 : 4);
    static constexpr int T = M / P, NW = T / 32;
    static constexpr int COLS = M / C, SEGT = COLS / P;      // columns; threads of a segment
    static constexpr bool SPLIT = COLS < T;
    static constexpr int LANES = SPLIT ? T / COLS : 1;       // lanes that share a column
    static constexpr int PER = SPLIT ? 1 : COLS / T;         // columns per thread
    static constexpr int NV = SPLIT ? P : PER * (C - 1);     // outer twiddles per thread
    static constexpr bool TABLES = M <= 2048;                // twiddles in shared memory
    using F = FftPlan<M, P>;
    static_assert(SEGT >= 2 || C == 1, "a segment spans threads");
    static_assert(LANES <= 4, "lane transforms of up to 4 points");
};

// Shared-memory placement of 16-byte element m: permuted inside every 128-byte row by
// higher bits, for conflict-free strided, unit-stride and per-thread contiguous access
template <int P>
__host__ __device__ constexpr int swzx(int m) {
    return P == 4 ? m ^ ((m >> 3) & 3) ^ ((m >> 2) & 4) : (P == 8 ? m ^ ((m >> 3) & 7) : m ^ ((m >> 4) & 7));
}
template <int P>
__device__ __forceinline__ int swzx_at(int s0, int k) { return (s0 ^ (swzx<P>(k) & 7)) + (k & ~7); }

template <typename R, int M, int C>
struct SmemX {
    using cplx = typename Num<R>::cplx;
    using SH = ShapeX<M, C>;
    static constexpr size_t off_x = 0;                                          // transform buffer
    static constexpr size_t off_g = off_x + sizeof(cplx) * M;                   // clusters: columns
    static constexpr size_t off_d = off_g + (C > 1 ? sizeof(cplx) * M : 0);     // per-mode dispersion factor
    static constexpr size_t off_tw = off_d + sizeof(cplx) * M;                  // pass twiddles
    static constexpr size_t off_xtw = off_tw + (SH::TABLES ? sizeof(cplx) * SH::F::TW : 0);   // outer twiddles
    static constexpr size_t off_edge = off_xtw + (SH::TABLES && C > 1 ? sizeof(cplx) * SH::NV * SH::T : 0);
    static constexpr size_t off_halo = off_edge + sizeof(cplx) * 4 * SH::NW;    // [parity][first, last][warp]
    // E and increment of every segment's 4 halo points; field and carrier of the end threads' two
    static constexpr size_t off_bar = off_halo + (C > 1 ? sizeof(cplx) * 16 * C : 0);
    static constexpr size_t off_red = off_bar + sizeof(uint64_t) * 4;
    // absorber factors of the threads that have one (a quarter of them: the absorber spans
    // [6/16, 10/16] of the window in every variant): [point][thread]
    static constexpr int SLOTS = SH::T / 4 + 2;
    static constexpr size_t off_abc = (off_red + sizeof(int) * (2 * SH::NW + 2 * 16 + 8) + 15) & ~size_t(15);
    static constexpr size_t bytes = off_abc + sizeof(typename Num<R>::real) * SH::P * SLOTS;
    static_assert(bytes <= 232448 - 288, "shared memory of one CTA");
};

// ---------------------------------------------------------------------------
// small DFTs in registers (radix-2 stages, decimation in frequency; register q ends
// holding output bitrev(q)) and their exact-order reverse; INV: conjugate twiddles.
// w16: W_16^m, m < 8.
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ typename Num<R>::cplx rotx(typename Num<R>::cplx v, int m16, bool inv,
                                                      const typename Num<R>::cplx* w16) {
    using X = Num<R>;
    if (m16 == 0) return v;
    if (m16 == 4) return inv ? X::mul_i(v) : X::mul_mi(v);
    return inv ? X::mulc(v, w16[m16]) : X::mul(v, w16[m16]);
}
template <typename R, int K>
__device__ __forceinline__ void dftx(typename Num<R>::cplx* v, const typename Num<R>::cplx* w16) {
    using X = Num<R>;
#pragma unroll
    for (int hr = K / 2; hr >= 1; hr >>= 1) {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            if (q & hr) continue;
            const typename X::cplx a = v[q], b = v[q + hr];
            v[q] = X::add(a, b);
            v[q + hr] = rotx<R>(X::sub(a, b), (q & (hr - 1)) * (K / (2 * hr)) * (16 / K), false, w16);
        }
    }
}
template <typename R, int K>
__device__ __forceinline__ void dftx_inv(typename Num<R>::cplx* v, const typename Num<R>::cplx* w16) {
    using X = Num<R>;
#pragma unroll
    for (int hr = 1; hr <= K / 2; hr <<= 1) {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            if (q & hr) continue;
            const typename X::cplx a = v[q];
            const typename X::cplx b = rotx<R>(v[q + hr], (q & (hr - 1)) * (K / (2 * hr)) * (16 / K), true, w16);
            v[q] = X::add(a, b);
            v[q + hr] = X::sub(a, b);
        }
    }
}

// ---------------------------------------------------------------------------
// M-point transform in shared memory, the scheme of ofx_fft.cuh in R.  The passes are
// loops over one body each: unrolled, a float-float attempt was over 100 KB of
// straight-line code and waited on instruction fetch.
// ---------------------------------------------------------------------------
template <typename R, int M, int C>
struct FftX {
    using X = Num<R>;
    using cplx = typename X::cplx;
    using SH = ShapeX<M, C>;
    using F = typename SH::F;
    static constexpr int P = SH::P;
    cplx* buf;
    const cplx* tw;          // shared-memory pass twiddles (TABLES)
    const cplx* wn;          // W_N, global
    const cplx* w16;
    int t;

    // twiddle of register q in pass ps (blocks of M >> (ps RB) points)
    __device__ __forceinline__ cplx twiddle(int ps, int q, int off) const {
        const int LR = (M >> (ps * F::RB)) / P;
        if constexpr (SH::TABLES) {
            // entries before pass ps: (P - 1)/P (M + M/P + ...) = M - (M >> ps RB)
            return tw[M - (M >> (ps * F::RB)) + (q - 1) * LR + off];
        } else {
            return wn[(size_t)((off * brev4(q, F::RB)) << (ps * F::RB)) * C];
        }
    }
    __device__ __forceinline__ void load_own(cplx (&v)[P]) const {
        const int s0 = swzx<P>(P * t);
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = buf[swzx_at<P>(s0, j)];
    }
    __device__ __forceinline__ void store_own(cplx* b, const cplx (&v)[P]) const {
        const int s0 = swzx<P>(P * t);
#pragma unroll
        for (int j = 0; j < P; ++j) b[swzx_at<P>(s0, j)] = v[j];
    }
    static __device__ __forceinline__ void sync(int group) {
        if (group <= 32) __syncwarp();
        else __syncthreads();
    }
    __device__ __forceinline__ void forward(cplx (&v)[P]) const {
#pragma unroll 1
        for (int ps = 0; ps < F::NP - 1; ++ps) {
            const int LR = (M >> (ps * F::RB)) / P, off = t & (LR - 1), base = (t - off) * P + off;
#pragma unroll
            for (int q = 0; q < P; ++q) v[q] = buf[swzx<P>(base + q * LR)];
            dftx<R, P>(v, w16);
#pragma unroll
            for (int q = 1; q < P; ++q) v[q] = X::mul(v[q], twiddle(ps, q, off));
#pragma unroll
            for (int q = 0; q < P; ++q) buf[swzx<P>(base + q * LR)] = v[q];
            sync(LR);
        }
        load_own(v);
#pragma unroll
        for (int u = 0; u < P / F::LAST; ++u) dftx<R, F::LAST>(v + u * F::LAST, w16);
    }
    // v[q] returns point t + q M/P
    __device__ __forceinline__ void inverse(cplx (&v)[P]) const {
#pragma unroll
        for (int u = 0; u < P / F::LAST; ++u) dftx_inv<R, F::LAST>(v + u * F::LAST, w16);
        store_own(buf, v);
        sync(F::L(F::NP - 2) / P);
#pragma unroll 1
        for (int ps = F::NP - 2; ps >= 0; --ps) {
            const int LR = (M >> (ps * F::RB)) / P, off = t & (LR - 1), base = (t - off) * P + off;
#pragma unroll
            for (int q = 0; q < P; ++q) v[q] = buf[swzx<P>(base + q * LR)];
#pragma unroll
            for (int q = 1; q < P; ++q) v[q] = X::mulc(v[q], twiddle(ps, q, off));
            dftx_inv<R, P>(v, w16);
            if (ps > 0) {
#pragma unroll
                for (int q = 0; q < P; ++q) buf[swzx<P>(base + q * LR)] = v[q];
                sync(LR * P);
            }
        }
    }
};

// 16-byte values into a peer's shared memory, counted on its mbarrier
template <typename V>
__device__ __forceinline__ void st_async16(uint32_t addr, V v, uint32_t bar) {
    static_assert(sizeof(V) == 16, "16-byte values");
    uint32_t w[4];
    memcpy(w, &v, 16);
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(bar) : "memory");
}
template <typename V>
__device__ __forceinline__ V shfl16(V v, int src, bool up, bool down, int mask) {
    uint32_t w[4];
    memcpy(w, &v, 16);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = up ? __shfl_up_sync(0xffffffffu, w[i], src)
                  : (down ? __shfl_down_sync(0xffffffffu, w[i], src) : __shfl_xor_sync(0xffffffffu, w[i], mask));
    memcpy(&v, w, 16);
    return v;
}

// Error class of one point from E and E - A1: pct = 100 |E - A1| / (|E| + 1) in
// FP64 (as the FP64 oracle), MEX rule (points with |E| = 0 skipped; >= maxErr,
// else >= minErr) or NEE rule (> maxErr; >= minErr).
template <typename R, bool NEE>
__device__ __forceinline__ int classify_x(typename Num<R>::cplx e, typename Num<R>::cplx d, double maxE,
                                          double minE) {
    const double2 ed = Num<R>::to_d(e), dd = Num<R>::to_d(d);
    const double ae = hypot(ed.x, ed.y);
    const double pct = 100.0 * hypot(dd.x, dd.y) / (ae + 1.0);
    int bits = 0;
    if (NEE) {
        if (pct > maxE) bits |= 1;
        if (pct >= minE) bits |= 2;
    } else if (ae > 0.0) {
        if (pct >= maxE) bits |= 1;
        else if (pct >= minE) bits |= 2;
    }
    if (!Num<R>::finite(e)) bits |= 4;
    return bits;
}

// OR of the classes of a thread's points.  FP32 magnitudes (of E and of K2 - K1, which
// is 2 (E - A1) to the working precision) decide where the largest error is 1e-5
// (relative) away from both thresholds and below the upper one; everything else goes
// through the FP64 classes, so every decision is FP64's.  Two FP64 hypot and a division
// a point were a third of the FP64 kernel's arithmetic.
template <typename R, bool NEE, int P>
__device__ __forceinline__ int classify_points(const typename Num<R>::cplx (&e)[P], const typename Num<R>::cplx (&d2)[P],
                                               const typename Num<R>::cplx (&a1)[P], const Bounds& B, double maxE,
                                               double minE) {
    using X = Num<R>;
    float qmax = 0.f, emin = 3e38f, sum = 0.f;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const float2 em = X::abs32(e[j]), dm = X::abs32(d2[j]);
        const float e2 = fmaf(em.x, em.x, em.y * em.y), dd = fmaf(dm.x, dm.x, dm.y * dm.y);
        const float r = rcp_fast(sqrt_fast(e2) + 1.f);
        qmax = fmaxf(qmax, dd * r * r);
        emin = fminf(emin, e2);
        sum += e2;
    }
    const bool low = qmax < B.qlo0, high = qmax > B.qlo1;
    if (sum < 1e30f && qmax < B.qhi && (low || (high && (NEE || emin > 1e-30f)))) return high ? 2 : 0;
    int bits = 0;
#pragma unroll
    for (int j = 0; j < P; ++j) bits |= classify_x<R, NEE>(e[j], X::sub(e[j], a1[j]), maxE, minE);
    return bits;
}

// ---------------------------------------------------------------------------
// the kernel: layout, exchange steps A to D and their ordering as pass_kernel
// (ofx_pass.cuh), in R
// ---------------------------------------------------------------------------
template <typename R, int M, int C, bool NEE>
__global__ void __launch_bounds__(M / ShapeX<M, C>::P, 1)
passx_kernel(const PulseX* __restrict__ pulses, XTables<R> tabs, KernelCfg cfg) {
    using X = Num<R>;
    using cplx = typename X::cplx;
    using real = typename X::real;
    using SH = ShapeX<M, C>;
    constexpr int T = SH::T, P = SH::P, COLS = SH::COLS, NW = SH::NW;
    constexpr int N = M * C, LOG2M = ilog2(M);
    using SM = SmemX<R, M, C>;
    extern __shared__ __align__(16) unsigned char smem[];
    cplx* bufX = reinterpret_cast<cplx*>(smem + SM::off_x);
    cplx* bufG = reinterpret_cast<cplx*>(smem + SM::off_g);
    cplx* D_s = reinterpret_cast<cplx*>(smem + SM::off_d);
    cplx* tw_s = reinterpret_cast<cplx*>(smem + SM::off_tw);
    cplx* xtw_s = reinterpret_cast<cplx*>(smem + SM::off_xtw);
    cplx* edge = reinterpret_cast<cplx*>(smem + SM::off_edge);
    cplx* halo_e = reinterpret_cast<cplx*>(smem + SM::off_halo);
    cplx* halo_d = halo_e + 4 * C;
    int* red = reinterpret_cast<int*>(smem + SM::off_red);
    int* dead = red + 2 * NW + 2 * 16;
    real* abc_s = reinterpret_cast<real*>(smem + SM::off_abc);
    __shared__ PulseX sP;
    __shared__ cplx w16[8];
    __shared__ int slots;
    __shared__ unsigned long long grid_last[3];

    const int t = threadIdx.x;
    const int c = (C > 1) ? (int)cg::this_cluster().block_rank() : 0;
    const int p = blockIdx.x / C;
    const cplx* __restrict__ wn = tabs.wn;
    if (t == 0) {
        sP = pulses[p];
        dead[0] = dead[kTold] = dead[kBars] = dead[kOut] = dead[kVerdict] = 0;
        slots = 0;
        for (int i = 0; i < 3; ++i) grid_last[i] = 0;
    }
    if (t < 8) w16[t] = wn[(size_t)t * (N / 16)];
    __syncthreads();
    const PulseX& Pd = sP;
    const FftX<R, M, C> fft{bufX, tw_s, wn, w16, t};

    // ---- prologue: twiddle tables, barriers, field, carrier, absorber, z-phasors ----
    if constexpr (SH::TABLES) {
        using F = typename SH::F;
        int o = 0;
#pragma unroll 1
        for (int ps = 0; ps < F::NP - 1; ++ps) {
            const int L = M >> (ps * F::RB), LR = L / P;
#pragma unroll 1
            for (int i = t; i < (P - 1) * LR; i += T) {
                const int q = i / LR + 1, off = i % LR;
                tw_s[o + i] = wn[(size_t)(off * bitrev(q, F::RB) * (M / L)) * C];
            }
            o += (P - 1) * LR;
        }
    }
    // outer twiddle i of this thread: W_N^{n2 k1}; k1 of a register of the column DFT
    auto outer_k = [&](int i) {
        if constexpr (SH::SPLIT) return brev4(i, ilog2(P)) + P * brev4(t % SH::LANES, ilog2(SH::LANES));
        else return brev4(i % (C > 1 ? C - 1 : 1) + 1, ilog2(C));
    };
    auto outer = [&](int i) -> cplx {
        if constexpr (SH::TABLES) return xtw_s[i * T + t];
        const int n2 = c * COLS + (SH::SPLIT ? t / SH::LANES : t * SH::PER + i / (C > 1 ? C - 1 : 1));
        return wn[(size_t)n2 * outer_k(i)];
    };
    cplx inner[SH::SPLIT ? P : 1];            // W_C^{lane ka}
    if constexpr (C > 1) {
        if constexpr (SH::TABLES) {
#pragma unroll 1
            for (int i = 0; i < SH::NV; ++i) {
                const int n2 = c * COLS + (SH::SPLIT ? t / SH::LANES : t * SH::PER + i / (C - 1));
                xtw_s[i * T + t] = wn[(size_t)n2 * outer_k(i)];
            }
        }
        if constexpr (SH::SPLIT) {
#pragma unroll
            for (int r = 0; r < P; ++r)
                inner[r] = wn[(size_t)((t % SH::LANES) * brev4(r, ilog2(P)) % C) * (N / C)];
        }
    }
    constexpr bool LOCAL = C <= 4;
    constexpr int kAll = (int)sizeof(cplx) * (LOCAL ? M - COLS : M);
    constexpr int kBytesA = 4 * (C - 1) + 64 * C, kBytesD = 64 * C;
    const uint32_t bars = smem_u32(smem + SM::off_bar);
    const uint32_t bar_a = bars, bar_b = bars + 8, bar_c = bars + 16, bar_d = bars + 24;
    if (C > 1 && t == 0) {
        for (int i = 0; i < 4; ++i) bar_init(bars + 8 * i);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_arm(bar_a, kBytesA);
        bar_arm(bar_b, kAll);
        bar_arm(bar_c, kAll);
        bar_arm(bar_d, kBytesD);
    }
    uint32_t ph_a = 0, ph_x = 0;
    const int seg = t / SH::SEGT, tin = t % SH::SEGT;
    const int i0 = seg * M + c * COLS + P * tin;             // this thread's first point
    const bool lend = C > 1 && tin == 0, rend = C > 1 && tin == SH::SEGT - 1;
    auto carrier = [&](int i) {
        return X::from(turn_unit_d(Pd.tau_theta * (uint64_t)(long long)time_index(i, N, cfg.time_mode)));
    };
    auto absorber = [&](int i) {
        if (cfg.abc_mode == ABC_NEE) {                       // NEE_CPU.m:114-121
            const int it = (i < N / 2) ? i : i - N;
            const double range = (double)(N - 1) * Pd.dt, a2t = fabs(2.0 * (double)it * Pd.dt);
            if (!(range - a2t < 0.25 * range)) return 1.0;
            const double sh = 1.0 / cosh(24.0 * (1.0 - a2t / range));
            return 1.0 - sh * sh;
        }
        if (cfg.abc_mode == ABC_NONE || !(i > 6 * (N / 16) && i < 10 * (N / 16))) return 1.0;
        if (cfg.abc_mode == ABC_HARD) return 0.0;            // OPO_CUDA_BATCH_XTAL.cu:105-137
        const double g = cosh((48.0 / (double)N) * fabs((double)i - (double)N / 2.0));
        return 1.0 - 1.0 / (g * g);
    };
    cplx a[P], cph[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        a[j] = X::from(Pd.E_in[i0 + j]);
        cph[j] = carrier(i0 + j);
    }
    // The absorber's factors, kept: an FP64 cosh and a division per point in every attempt
    // cost the threads that have some 2 to 13 us (us per attempt, recomputed and kept: FP64
    // 2^12 points 30.4 and 28.4, 2^16 213 and 203; float-float 2^14 20.2 and 17.5, 2^16 87
    // and 74).  The FP64 kernel of 2048 points per CTA is the exception (107 and 116).
    constexpr bool kKeep = !(std::is_same<R, double>::value && M == 2048);
    int absorb = -1;
    if (i0 + P > 6 * (N / 16) && i0 <= 10 * (N / 16) && cfg.abc_mode != ABC_NONE) {
        absorb = kKeep ? atomicAdd(&slots, 1) : 0;
        if constexpr (kKeep) {
#pragma unroll 1
            for (int j = 0; j < P; ++j) abc_s[j * SM::SLOTS + absorb] = X::rfrom(absorber(i0 + j));
        }
    }
    // the end threads' two halo points: hs[0..1] field, hs[2..3] carrier
    cplx* hs = halo_e + 8 * C + 4 * (2 * seg + (rend ? 1 : 0));
    if (lend || rend) {
        const int i1 = lend ? (i0 + N - 1) % N : (i0 + P) % N;
        const int i2 = lend ? (i0 + N - 2) % N : (i0 + P + 1) % N;
        hs[0] = X::from(Pd.E_in[i1]); hs[1] = X::from(Pd.E_in[i2]);
        hs[2] = carrier(i1); hs[3] = carrier(i2);
    }
    // z-carrier phasor of every z-sample of the pass, shared by the cluster's CTAs
    cplx* ztab = reinterpret_cast<cplx*>(Pd.ztab);
    for (int pz = c * T + t; pz < Pd.zcap; pz += C * T)
        ztab[pz] = X::from(turn_unit_d((uint64_t)0 - Pd.tau_z * (uint64_t)pz));
    if constexpr (C > 1) cg::this_cluster().sync(); else __syncthreads();

    const double h = Pd.h, sel = Pd.sel, Sd = (double)Pd.S;
    const double maxE = Pd.max_err, minE = Pd.min_err;
    const Bounds bounds(50.f, (float)maxE, (float)minE);
    constexpr double invN = 1.0 / (double)N;
    const int guard = cfg.guard;
    const int max_attempts = cfg.max_attempts_mul * (Pd.S + 16) + 64;
    const int nchunks = Pd.nchunks;
    const bool rec = (c == 0 && t == 0);
    const real csr = X::rfrom(Pd.c_shock);

    double k = NEE ? 1.0 : 0.0, stepprev = 4.0, stepmod = 4.0;
    long long q = 0;
    int s_cached = -1;
    int attempt = 0, n_acc = 0, n_rej = 0, status = 0, par = 0;

    // A^2 e + 2 |A|^2 conj(e) with e = carrier z: A conj(3 Re w + i Im w) with w = A e
    auto drive = [&](cplx s, cplx car, cplx zz) -> cplx {
        const cplx w = X::mul(s, X::mul(car, zz));
        return X::mulc(s, X::make(X::triple(X::re(w)), X::im(w)));
    };
    // K = -i hG (NL - i cs (NL[+1] - NL[-1]))
    auto k_of = [&](cplx nm, cplx n0, cplx np, real hg) -> cplx {
        return X::mul_mi(X::scale(X::sub_i(n0, X::sub(np, nm), csr), hg));
    };
    // the neighbours' adjacent drive values; hv: the halo point's (end threads)
    auto edges = [&](const cplx (&nl)[P], cplx hv, cplx& L, cplx& Rr) {
        L = shfl16(nl[P - 1], 1, true, false, 0);
        Rr = shfl16(nl[0], 1, false, true, 0);
        if constexpr (SH::SEGT > 32) {
            const int w = t >> 5, lane = t & 31;
            cplx* e = edge + par * 2 * NW;
            if (lane == 0) e[w] = nl[0];
            if (lane == 31) e[NW + w] = nl[P - 1];
            __syncthreads();
            if (lane == 0) L = e[NW + (w > 0 ? w - 1 : NW - 1)];
            if (lane == 31) Rr = e[w < NW - 1 ? w + 1 : 0];
        }
        if (lend) L = hv;
        if (rend) Rr = hv;
        par ^= 1;
    };
    auto zphasor = [&](long long pz) -> cplx {
        return pz < Pd.zcap ? ztab[pz] : X::from(turn_unit_d((uint64_t)0 - Pd.tau_z * (uint64_t)pz));
    };
    // a value into CTA r's buffer at element i (same place in every CTA)
    auto push = [&](cplx* b, int r, int i, cplx v, uint32_t bar) {
        if (LOCAL && r == c) {
            b[i] = v;
        } else {
            const uint32_t src = smem_u32(b), dst = cluster_addr(src, r);
            st_async16(dst + 16 * i, v, dst + (bar - src));
        }
    };
    // v: point `col` of this CTA's segment sg, if it is one of the segment's two first or
    // last points, into the neighbours' halo slots
    auto push_halo_x = [&](cplx* b, int sg, int col, cplx v, uint32_t bar) {
        if (col >= 2 && col < COLS - 2) return;
        const bool first = col < 2;
        const int slot = first ? 4 * seg_left<C>(sg, c) + 2 + col : 4 * seg_right<C>(sg, c) + col - (COLS - 2);
        const uint32_t src = smem_u32(b), dst = cluster_addr(src, first ? (c + C - 1) % C : (c + 1) % C);
        st_async16(dst + 16 * slot, v, dst + (bar - src));
    };

    for (int chunk = 0; chunk < nchunks; ++chunk) {
        if (!NEE) stepmod = stepprev;
        const double cend = (double)(chunk + 1) * sel;
        while (k < cend && (NEE ? k <= Sd : (!guard || k < Sd))) {
            if (attempt >= max_attempts) { status |= OPTIFAX_PULSE_ATTEMPT_LIMIT; goto done; }
            const int kidx = NEE ? (int)k - 1 : (int)k;
            const int krec = (int)k;
            const double kpos = NEE ? k - 1.0 : k;
            bool accepted = false;
            const real hg = X::rfrom((stepmod * h) * Pd.G[kidx]);
            cplx e[P];
            int bits;
            {
                cplx nl[P], k1[P], a1[P], d2[P], kh = X::zero();
#pragma unroll
                for (int j = 0; j < P; ++j) { a1[j] = a[j]; k1[j] = X::zero(); }
                // stage 0: K1 = f(A0) at z = k; stage 1: K2 = f(A1) at z = k + stepmod, with
                // A1 = A0 + (K1/2 + K1/2) (MEX) or A0 + K1 (NEE_CPU.m:73), the same value.
                // One body for both (code size).
#pragma unroll 1
                for (int st = 0; st < 2; ++st) {
                    const cplx z = zphasor((long long)(st ? kpos + stepmod : kpos));
#pragma unroll
                    for (int j = 0; j < P; ++j) nl[j] = drive(a1[j], cph[j], z);
                    cplx hv = X::zero(), L, Rr;
                    if (lend || rend) {      // drive of the adjacent halo point, and its K1
                        hv = drive(X::add(hs[0], kh), hs[2], z);
                        if (st == 0) {
                            const cplx n2 = drive(hs[1], hs[3], z), in = lend ? nl[0] : nl[P - 1];
                            kh = k_of(lend ? n2 : in, hv, lend ? in : n2, hg);
                        }
                    }
                    edges(nl, hv, L, Rr);
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        const cplx kk = k_of(j == 0 ? L : nl[j - 1], nl[j], j == P - 1 ? Rr : nl[j + 1], hg);
                        if (st == 0) {
                            k1[j] = kk;
                            a1[j] = X::add(a[j], kk);
                        } else {
                            d2[j] = kk;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    // E = A0 + (K2/2 + K1/2) (MEX) or (A0 + K1/2) + K2/2 (NEE_CPU.m:75)
                    e[j] = NEE ? X::add_half(X::add_half(a[j], k1[j]), d2[j]) : X::add_half(a[j], X::add(d2[j], k1[j]));
                    d2[j] = X::sub(d2[j], k1[j]);
                }
                // pct = 100 |E - A1| / (|E| + 1) (OPO_CUDA_BATCH_XTAL.cu:325-349; NEE_CPU.m:73-79)
                bits = classify_points<R, NEE, P>(e, d2, a1, bounds, maxE, minE);
            }
            if (absorb >= 0) {
#pragma unroll
                for (int j = 0; j < P; ++j)
                    e[j] = X::scale(e[j], kKeep ? abc_s[j * SM::SLOTS + absorb] : X::rfrom(absorber(i0 + j)));
            }
            fft.store_own(C > 1 ? bufG : bufX, e);
            if constexpr (C > 1) {
                if (lend || rend || P < 2) {
#pragma unroll
                    for (int j = 0; j < P; ++j) push_halo_x(halo_e, seg, P * tin + j, e[j], bar_a);
                }
            }
            int fl = combine_flags<NW, C>(bits, red, bar_a, ph_a, kBytesA, dead, grid_last, attempt, t, c, cfg);
            ph_a ^= 1;
            if (fl & kDead) goto done;
            if (fl & 4) status |= OPTIFAX_PULSE_NAN;

            if ((fl & 1) && stepmod > 1.0 && (NEE || (k - stepmod) > 0.0)) {
                if (rec && Pd.trace && attempt < Pd.trace_cap) {
                    Pd.trace[3 * attempt] = krec; Pd.trace[3 * attempt + 1] = (int)stepmod;
                    Pd.trace[3 * attempt + 2] = fl & 7;
                }
                ++n_rej;
                // the next attempt's flags and halos must not overtake this one's
                if constexpr (C > 1) {
                    count_bar(dead, t);
                    cg::this_cluster().sync();
                    if (peer_gone(dead)) goto done;
                }
                if (!NEE) k = k - stepmod;
                stepmod = stepmod - 1.0;
                stepprev = stepmod;
            } else {
                if (rec && Pd.trace && attempt < Pd.trace_cap) {
                    Pd.trace[3 * attempt] = krec; Pd.trace[3 * attempt + 1] = (int)stepmod;
                    Pd.trace[3 * attempt + 2] = (fl & 7) | 8;
                }
                ++n_acc;
                accepted = true;
                const int s_used = (int)stepmod;
                if (NEE) {
                    if (!(fl & 2)) stepmod = stepmod + 1.0;
                    if (k < Sd && k + stepmod > Sd) stepmod = Sd - k;
                } else if (k + stepmod >= cend && k < cend - 1.0) {
                    const double stepend = (cend - k) - 1.0;
                    stepprev = stepmod;
                    stepmod = stepend;
                } else {
                    if (!(fl & 2) && !(fl & 1) && (k + stepmod + 1.0) < cend - 1.0) stepmod = stepmod + 1.0;
                    stepprev = stepmod;
                }

                // ---- linear sub-step: A0 = IFFT(D FFT(E abc)) / N ----
                cplx v[P];
                if constexpr (C > 1) {
                    if (lend || rend) {
                        hs[0] = halo_e[4 * seg + (lend ? 1 : 2)];
                        hs[1] = halo_e[4 * seg + (lend ? 0 : 3)];
                    }
                    // C-point DFTs of the own columns, twiddle -> the blocks' owners
                    if constexpr (SH::SPLIT) {
                        const int l = t % SH::LANES, col = t / SH::LANES;
#pragma unroll
                        for (int i = 0; i < P; ++i) v[i] = bufG[swzx<P>((i * SH::LANES + l) * COLS + col)];
                        dftx<R, P>(v, w16);
#pragma unroll
                        for (int r = 1; r < P; ++r) v[r] = X::mul(v[r], inner[r]);
#pragma unroll
                        for (int hr = SH::LANES / 2; hr >= 1; hr >>= 1) {
                            const bool up = (l & hr) != 0, turn = SH::LANES == 4 && hr == 2 && (l & 1);
#pragma unroll
                            for (int i = 0; i < P; ++i) {
                                const cplx o = shfl16(v[i], 0, false, false, hr);
                                cplx d = up ? X::sub(o, v[i]) : X::add(v[i], o);
                                v[i] = up && turn ? X::mul_mi(d) : d;
                            }
                        }
#pragma unroll
                        for (int r = 0; r < P; ++r)
                            push(bufX, outer_k(r), swzx<P>(c * COLS + col), X::mul(v[r], outer(r)), bar_b);
                    } else {
#pragma unroll
                        for (int u = 0; u < SH::PER; ++u) {
                            cplx y[C];
#pragma unroll
                            for (int n1 = 0; n1 < C; ++n1) y[n1] = bufG[swzx<P>(n1 * COLS + t * SH::PER + u)];
                            dftx<R, C>(y, w16);
#pragma unroll
                            for (int r = 0; r < C; ++r) {
                                if (r > 0) y[r] = X::mul(y[r], outer(u * (C - 1) + r - 1));
                                push(bufX, brev4(r, ilog2(C)), swzx<P>(c * COLS + t * SH::PER + u), y[r], bar_b);
                            }
                        }
                    }
                }
                if (s_used != s_cached) {
                    // D_k = alpha_k^s exp(-i beta_k s) / N in FP64 (OPO_CUDA_BATCH_XTAL.cu:255-305)
#pragma unroll 1
                    for (int j = 0; j < P; ++j) {
                        const int kk = c + C * bitrev(P * t + j, LOG2M);
                        double sn, cn;
                        sincos(-Pd.beta[kk] * (double)s_used, &sn, &cn);
                        const double al = Pd.alpha[kk];
                        const double af = (al == 1.0) ? 1.0 : pow(al, (double)s_used);
                        D_s[j * T + t] = X::from(make_double2(cn * af * invN, sn * af * invN));   // 1/N: exact
                    }
                    s_cached = s_used;
                }
                if constexpr (C > 1) {
                    if constexpr (LOCAL) __syncthreads();
                    bar_next(bar_b, ph_x, kAll, dead, cfg.wait, t);
                }
                fft.forward(v);
#pragma unroll
                for (int j = 0; j < P; ++j) v[j] = X::mul(v[j], D_s[j * T + t]);
                fft.inverse(v);
                if constexpr (C > 1) {
                    // outputs (points t + q M/P of the block) -> their columns' owners; with more
                    // CTAs than points a thread does not add to every peer's bytes, which then
                    // say nothing about its reads of the transform buffer
                    if constexpr (C > P) __syncthreads();
#pragma unroll
                    for (int i = 0; i < P; ++i) {
                        const int m = t + i * T;
                        push(bufG, m / COLS, swzx<P>(c * COLS + m % COLS), v[i], bar_c);
                    }
                    if constexpr (LOCAL) __syncthreads();
                    bar_next(bar_c, ph_x, kAll, dead, cfg.wait, t);
                    // undo the twiddles, inverse C-point DFTs -> own points
                    if constexpr (SH::SPLIT) {
                        const int l = t % SH::LANES, col = t / SH::LANES;
#pragma unroll
                        for (int r = 0; r < P; ++r)
                            v[r] = X::mulc(bufG[swzx<P>(outer_k(r) * COLS + col)], outer(r));
#pragma unroll
                        for (int hr = 1; hr <= SH::LANES / 2; hr <<= 1) {
                            const bool up = (l & hr) != 0, turn = SH::LANES == 4 && hr == 2 && (l & 1);
#pragma unroll
                            for (int i = 0; i < P; ++i) {
                                if (up && turn) v[i] = X::mul_i(v[i]);
                                const cplx o = shfl16(v[i], 0, false, false, hr);
                                v[i] = up ? X::sub(o, v[i]) : X::add(v[i], o);
                            }
                        }
#pragma unroll
                        for (int r = 1; r < P; ++r) v[r] = X::mulc(v[r], inner[r]);
                        dftx_inv<R, P>(v, w16);
#pragma unroll
                        for (int i = 0; i < P; ++i) {
                            const int n1 = i * SH::LANES + l;
                            bufX[swzx<P>(n1 * COLS + col)] = v[i];
                            push_halo_x(halo_d, n1, col, v[i], bar_d);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < SH::PER; ++u) {
                            const int col = t * SH::PER + u;
                            cplx y[C];
#pragma unroll
                            for (int r = 0; r < C; ++r) {
                                y[r] = bufG[swzx<P>(brev4(r, ilog2(C)) * COLS + col)];
                                if (r > 0) y[r] = X::mulc(y[r], outer(u * (C - 1) + r - 1));
                            }
                            dftx_inv<R, C>(y, w16);
#pragma unroll
                            for (int n1 = 0; n1 < C; ++n1) {
                                bufX[swzx<P>(n1 * COLS + col)] = y[n1];
                                push_halo_x(halo_d, n1, col, y[n1], bar_d);
                            }
                        }
                    }
                    __syncthreads();
                    if (lend || rend) {
                        bar_next(bar_d, ph_x, kBytesD, dead, cfg.wait, t);
                        hs[0] = halo_d[4 * seg + (lend ? 1 : 2)];
                        hs[1] = halo_d[4 * seg + (lend ? 0 : 3)];
                    }
                    ph_x ^= 1;
                } else {
                    const int s0 = swzx<P>(t);
#pragma unroll
                    for (int i = 0; i < P; ++i) bufX[swzx_at<P>(s0, i * T)] = v[i];
                    __syncthreads();
                }
                fft.load_own(a);
                q += s_used;
            }
            ++attempt;
            if (!NEE || accepted) k = k + stepmod;
        }
    }
done:
    const bool gone = last_word<C>(dead);
#pragma unroll
    for (int j = 0; j < P; ++j) Pd.A_out[i0 + j] = X::to_d(a[j]);
    if (rec && Pd.stats) {
        optifax_pulse_stats st;
        st.attempts = attempt; st.accepted = n_acc; st.rejected = n_rej; st.status = status;
        st.z_steps = q; st.k_final = (float)k; st.stepmod_final = (float)stepmod; st.n_chunks = nchunks;
        st.reserved[0] = 1; st.reserved[1] = st.reserved[2] = 0;
        *Pd.stats = st;
    }
    if constexpr (C > 1) {
        if (!gone) cg::this_cluster().sync();        // no CTA leaves while a peer may still write its memory
    }
    end_lost<M, C>(dead, Pd.A_out, Pd.stats, cfg);
}

}  // namespace ofx
