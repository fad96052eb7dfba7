// ofx_fft.cuh -- in-shared-memory complex FFT of one CTA's M points with P points
// per thread (P = 4 or 8), for the FP32 crystal pass and the fibre kernel.
//
// Decimation in frequency: passes of radix P over blocks of length M, M/P, ...; the
// last pass has the remaining radix.  In a pass over blocks of length L every thread
// owns one butterfly: y_q = W_L^{off r} DFT_P(x[off + q L/P])_r with r = bitrev(q), so
// the forward transform leaves the spectrum in bit-reversed slot order and the inverse
// undoes it, multiplying by the exact reciprocal conj(w)(1 + d) of every forward
// twiddle.  The last forward and the first inverse pass act on the same registers
// (thread t holds slots P t .. P t + P - 1).  Unnormalised: forward then inverse
// multiplies by M.
//
// The outer twiddles sit in shared memory: (c, s) as [pass][q - 1][off] and the
// reciprocals' d = 1/|w|^2 - 1 as [pass][off][P], read as vectors.
//
// Eight points per thread instead of sixteen: twice the warps hide the latency of the
// fixed-latency chains and shared-memory round trips that bound the pass (two warps per
// scheduler issued on half of the cycles), for one more pass through shared memory at
// 4096 points.
#pragma once
#include "ofx_common.cuh"

namespace ofx {

// Points per thread of a CTA with M points
template <int M>
constexpr int kPoints = (M >= 2048) ? 8 : 4;

__host__ __device__ constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x / 2); }

template <int M, int P>
struct FftPlan {
    static constexpr int T = M / P, RB = ilog2(P), BITS = ilog2(M);
    static constexpr int NP = (BITS + RB - 1) / RB;                 // passes
    static constexpr int LAST = 1 << (BITS - (NP - 1) * RB);        // radix of the last pass
    static constexpr int L(int p) { return M >> (p * RB); }         // block length of pass p
    static constexpr int tw_off(int p) { return p == 0 ? 0 : tw_off(p - 1) + (P - 1) * (L(p - 1) / P); }
    static constexpr int td_off(int p) { return p == 0 ? 0 : td_off(p - 1) + L(p - 1); }
    static constexpr int TW = tw_off(NP - 1);                       // float2 entries
    static constexpr int TD = td_off(NP - 1);                       // d entries
};

// Shared-memory placement of point m: 16-byte pairs are permuted inside every 128-byte
// row by higher bits of m, so that the strided accesses of every pass, the per-thread
// contiguous accesses (16-byte vectors) and the unit-stride ones are free of bank
// conflicts without padding.  swz is linear over XOR.
__host__ __device__ constexpr int swz(int m) { return m ^ (((m >> 4) & 3) << 1) ^ ((m >> 3) & 8); }

// swz(base + k) for s0 = swz(base) where base has zeros in the bits of the constant k
__device__ __forceinline__ int swz_at(int s0, int k) { return (s0 ^ (swz(k) & 15)) + (k & ~15); }

// W_16^m = exp(-2 pi i m / 16), m = 0..7, rounded to FP32; d = 1/|w|^2 - 1
__device__ __forceinline__ float w16c(int m) {
    constexpr float c[8] = {1.0f, 0.9238795042037964f, 0.7071067690849304f, 0.3826834261417389f,
                            0.0f, -0.3826834261417389f, -0.7071067690849304f, -0.9238795042037964f};
    return c[m];
}
__device__ __forceinline__ float w16s(int m) {
    constexpr float s[8] = {0.0f, -0.3826834261417389f, -0.7071067690849304f, -0.9238795042037964f,
                            -1.0f, -0.9238795042037964f, -0.7071067690849304f, -0.3826834261417389f};
    return s[m];
}
__device__ __forceinline__ float w16d(int m) {
    constexpr float d[8] = {0.0f, 5.7068572090201997e-08f, 3.422854177870249e-08f, 5.7068572090201997e-08f,
                            0.0f, 5.7068572090201997e-08f, 3.422854177870249e-08f, 5.7068572090201997e-08f};
    return d[m];
}

__device__ __forceinline__ int brev4(int q, int bits) {
    // bit reversal of q within `bits` (<= 4) bits, compile-time foldable
    int r = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if (b < bits && (q & (1 << b))) r |= 1 << (bits - 1 - b);
    return r;
}

// Small DFTs in registers with packed additions: radix-2 stages, forward decimation in
// frequency (register q ends holding output bitrev(q)), the inverse its exact reverse
// (every constant's exact reciprocal).  m16: exponent of W_16.
__device__ __forceinline__ float2 rot_fwd(float2 v, int m16) {
    if (m16 == 0) return v;
    if (m16 == 4) return make_float2(v.y, -v.x);
    if (m16 == 2 || m16 == 6) {                            // c (1 - i), c (-1 - i)
        const float2 t = mul2(v, dup2(w16c(2)));
        return m16 == 2 ? make_float2(t.x + t.y, t.y - t.x) : make_float2(t.y - t.x, -(t.x + t.y));
    }
    return cmul(v, make_float2(w16c(m16), w16s(m16)));
}
__device__ __forceinline__ float2 rot_inv(float2 v, int m16) {
    if (m16 == 0) return v;
    if (m16 == 4) return make_float2(-v.y, v.x);
    float2 u;
    if (m16 == 2 || m16 == 6) {
        const float2 t = mul2(v, dup2(w16c(2)));
        u = m16 == 2 ? make_float2(t.x - t.y, t.y + t.x) : make_float2(-(t.x + t.y), t.x - t.y);
    } else {
        u = cmulc(v, make_float2(w16c(m16), w16s(m16)));
    }
    return cfma1(u, w16d(m16), u);
}
template <int R>
__device__ __forceinline__ void dftp(float2* v) {
#pragma unroll
    for (int hr = R / 2; hr >= 1; hr >>= 1) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (q & hr) continue;
            const float2 a = v[q], b = v[q + hr];
            v[q] = add2(a, b);
            v[q + hr] = rot_fwd(sub2(a, b), (q & (hr - 1)) * (R / (2 * hr)) * (16 / R));
        }
    }
}
template <int R>
__device__ __forceinline__ void dftp_inv(float2* v) {
#pragma unroll
    for (int hr = 1; hr <= R / 2; hr <<= 1) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (q & hr) continue;
            const float2 a = v[q], t = rot_inv(v[q + hr], (q & (hr - 1)) * (R / (2 * hr)) * (16 / R));
            v[q] = add2(a, t);
            v[q + hr] = sub2(a, t);
        }
    }
}

// this thread's P contiguous points (16-byte vectors)
template <int P>
__device__ __forceinline__ void load_own(const float2* buf, int t, float2 (&v)[P]) {
    const int s0 = swz(P * t);
#pragma unroll
    for (int j = 0; j < P; j += 2) {
        const float4 w = *reinterpret_cast<const float4*>(buf + (s0 ^ j));
        v[j] = make_float2(w.x, w.y);
        v[j + 1] = make_float2(w.z, w.w);
    }
}
template <int P>
__device__ __forceinline__ void store_own(float2* buf, int t, const float2 (&v)[P]) {
    const int s0 = swz(P * t);
#pragma unroll
    for (int j = 0; j < P; j += 2)
        *reinterpret_cast<float4*>(buf + (s0 ^ j)) = make_float4(v[j].x, v[j].y, v[j + 1].x, v[j + 1].y);
}

// v / w for w = (c, s) with reciprocal correction d
__device__ __forceinline__ float2 mul_recip(float2 v, float2 w, float d) {
    const float2 t = cmulc(v, w);
    return cfma1(t, d, t);
}

// Barrier between two passes whose data stay inside aligned groups of `group` threads
template <int GROUP>
__device__ __forceinline__ void pass_sync() {
    if constexpr (GROUP <= 32) __syncwarp();
    else __syncthreads();
}

// Fill the twiddle tables from the quarter-period table of W_M (global memory).
template <int M, int P>
__device__ __forceinline__ void fft_tables(float2* tw, float* td, const Twiddle* quad, int t) {
    using F = FftPlan<M, P>;
#pragma unroll 1
    for (int p = 0; p < F::NP - 1; ++p) {
        const int L = M >> (p * F::RB), LR = L / P;
        int o = 0, od = 0;
        for (int i = 0; i < p; ++i) { o += (P - 1) * ((M >> (i * F::RB)) / P); od += M >> (i * F::RB); }
#pragma unroll 1
        for (int i = t; i < L; i += F::T) {
            const int q = i / LR, off = i - q * LR;
            const int r = bitrev(q, F::RB);
            const Twiddle w = quad_tw<M>(quad, off * r * (M / L));
            if (q > 0) tw[o + (q - 1) * LR + off] = make_float2(w.c, w.s);
            td[od + off * P + q] = w.d;
        }
    }
}

// One forward pass; LOAD: from buf, else v holds points base + q L/P of the block.
template <int M, int P, int PASS, bool LOAD = true>
__device__ __forceinline__ void fftp_fwd(float2* buf, const float2* tw, int t, float2 (&v)[P]) {
    using F = FftPlan<M, P>;
    constexpr int L = F::L(PASS), LR = L / P;
    const int off = t & (LR - 1), s0 = swz((t - off) * P + off);
    if constexpr (LOAD) {
#pragma unroll
        for (int q = 0; q < P; ++q) v[q] = buf[swz_at(s0, q * LR)];
    }
    dftp<P>(v);
#pragma unroll
    for (int q = 1; q < P; ++q) v[q] = cmul(v[q], tw[F::tw_off(PASS) + (q - 1) * LR + off]);
#pragma unroll
    for (int q = 0; q < P; ++q) buf[swz_at(s0, q * LR)] = v[q];
}

// One inverse pass; on return v[q] holds points base + q L/P of the block.
template <int M, int P, int PASS>
__device__ __forceinline__ void fftp_inv(const float2* buf, const float2* tw, const float* td, int t,
                                         float2 (&v)[P], int& s0) {
    using F = FftPlan<M, P>;
    constexpr int L = F::L(PASS), LR = L / P;
    const int off = t & (LR - 1);
    s0 = swz((t - off) * P + off);
    float d[P];
#pragma unroll
    for (int q = 0; q < P; q += 4) {
        const float4 w = *reinterpret_cast<const float4*>(td + F::td_off(PASS) + off * P + q);
        d[q] = w.x; d[q + 1] = w.y; d[q + 2] = w.z; d[q + 3] = w.w;
    }
#pragma unroll
    for (int q = 0; q < P; ++q) v[q] = buf[swz_at(s0, q * LR)];
#pragma unroll
    for (int q = 1; q < P; ++q) v[q] = mul_recip(v[q], tw[F::tw_off(PASS) + (q - 1) * LR + off], d[q]);
    dftp_inv<P>(v);
}

template <int M, int P, int PASS>
__device__ __forceinline__ void fftp_forward_passes(float2* buf, const float2* tw, int t) {
    using F = FftPlan<M, P>;
    if constexpr (PASS < F::NP - 1) {
        float2 v[P];
        fftp_fwd<M, P, PASS>(buf, tw, t, v);
        pass_sync<F::L(PASS) / P>();
        fftp_forward_passes<M, P, PASS + 1>(buf, tw, t);
    }
}

// The last forward pass: v[j] returns slot P t + j
template <int M, int P>
__device__ __forceinline__ void fftp_forward_last(const float2* buf, int t, float2 (&v)[P]) {
    using F = FftPlan<M, P>;
    load_own<P>(buf, t, v);
#pragma unroll
    for (int u = 0; u < P / F::LAST; ++u) dftp<F::LAST>(v + u * F::LAST);
}

// Forward transform of buf (complete and visible); v[j] returns slot P t + j.
template <int M, int P>
__device__ __forceinline__ void fftp_forward(float2* buf, const float2* tw, int t, float2 (&v)[P]) {
    fftp_forward_passes<M, P, 0>(buf, tw, t);
    fftp_forward_last<M, P>(buf, t, v);
}

// Forward transform of v[q] = point t + q M/P, as fftp_inverse leaves them: the first
// pass works on the registers, through which a point-wise step between an inverse and a
// forward transform costs no shared-memory round trip.  buf is scratch whose previous
// reads by other threads are ordered before (fftp_inverse of the same buffer is).
template <int M, int P>
__device__ __forceinline__ void fftp_forward_regs(float2* buf, const float2* tw, int t, float2 (&v)[P]) {
    using F = FftPlan<M, P>;
    fftp_fwd<M, P, 0, false>(buf, tw, t, v);
    pass_sync<F::L(0) / P>();
    fftp_forward_passes<M, P, 1>(buf, tw, t);
    fftp_forward_last<M, P>(buf, t, v);
}

template <int M, int P, int PASS>
__device__ __forceinline__ void fftp_inverse_passes(float2* buf, const float2* tw, const float* td, int t) {
    using F = FftPlan<M, P>;
    if constexpr (PASS > 0) {
        float2 v[P];
        int s0;
        fftp_inv<M, P, PASS>(buf, tw, td, t, v, s0);
#pragma unroll
        for (int q = 0; q < P; ++q) buf[swz_at(s0, q * (F::L(PASS) / P))] = v[q];
        pass_sync<F::L(PASS - 1) / P>();
        fftp_inverse_passes<M, P, PASS - 1>(buf, tw, td, t);
    }
}

// Inverse of fftp_forward up to its last pass: on return v[q] holds points
// t + q M/P (q < P) of the unnormalised inverse transform.  Each thread writes only
// its own slots before the first barrier, so none is needed on entry.
template <int M, int P>
__device__ __forceinline__ void fftp_inverse(float2* buf, const float2* tw, const float* td, int t,
                                             float2 (&v)[P]) {
    using F = FftPlan<M, P>;
#pragma unroll
    for (int u = 0; u < P / F::LAST; ++u) dftp_inv<F::LAST>(v + u * F::LAST);
    store_own<P>(buf, t, v);
    pass_sync<F::L(F::NP - 2) / P>();
    fftp_inverse_passes<M, P, F::NP - 2>(buf, tw, td, t);
    int s0;
    fftp_inv<M, P, 0>(buf, tw, td, t, v, s0);
}

}  // namespace ofx
