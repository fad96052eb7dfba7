// ofx_common.cuh -- device helpers shared by the crystal-pass kernels.
//
// Complex arithmetic on float2, the fixed-point phase representation used to
// keep every accumulated phase exact to FP64 precision without FP64 work in
// the inner loops, and the twiddle-table entry layout.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ofx {

// Packed FP32 pairs (add/sub/mul/fma.f32x2): two IEEE operations per issued
// instruction, each rounded as its scalar form.  The kernels here are bound by issue
// slots and latency, not by the FMA pipe.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long x, y, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}

// a s + b
__device__ __forceinline__ float2 cfma1(float2 a, float s, float2 b) { return fma2(a, dup2(s), b); }

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// A phase in turns held as an unsigned 64-bit fixed-point fraction
// (2^64 == one turn).  Products of a per-unit phase with an integer position
// wrap modulo one turn exactly, so z-positions up to 2^32 keep the phase
// exact to ~1e-19 turns.  turn_to_unit returns exp(2 pi i u / 2^64) with the
// top 24 bits evaluated by sincospif and the remaining bits applied as a
// first-order rotation (|remainder| < 2 pi 2^-24 rad), accurate to ~1 ulp.
__device__ __forceinline__ float2 turn_to_unit(uint64_t u) {
    int32_t hi = (int32_t)(u >> 32);
    int32_t a = hi >> 8;                               // top 24 bits, signed
    float x = (float)a * 0x1p-23f;                     // half-turns in [-1, 1)
    float s, c;
    sincospif(x, &s, &c);
    uint32_t r24 = (uint32_t)((u << 24) >> 40);       // next 24 bits
    float d = (float)r24 * (0x1p-48f * 6.28318530717958647692f);
    return make_float2(fmaf(-s, d, c), fmaf(c, d, s));
}

// Twiddle entry: w = (c, s) ~ exp(-2 pi i e / n) rounded to FP32, and
// d = 1/|w|^2 - 1 evaluated in FP64.  The inverse transform multiplies by
// conj(w) (1 + d), the exact reciprocal of w up to one rounding, so a forward
// plus inverse transform carries no systematic per-mode gain.
struct __align__(16) Twiddle { float c, s, d, pad; };

// W_M^x for 0 <= x < M from the quarter-period table q[y] = W_M^y, y < M/4
// (kept in shared memory): x = k M/4 + y gives W_M^y (-i)^k, a swap and sign
// changes, so the value and its d are those of a full table.
template <int M>
__device__ __forceinline__ Twiddle quad_tw(const Twiddle* q, int x) {
    const Twiddle w = q[x & (M / 4 - 1)];
    const int k = (x / (M / 4)) & 3;
    float c = (k & 1) ? w.s : w.c;
    float s = (k & 1) ? -w.c : w.s;
    if (k & 2) { c = -c; s = -s; }
    return Twiddle{c, s, w.d, 0.f};
}

// 1/|w|^2 - 1 for a computed |w| ~ 1.  g = |w|^2 - 1 is formed without
// rounding error beyond the last add (products split by fma; the subtractions
// are exact by Sterbenz's lemma), then 1/(1 + g) - 1 = -g + g^2 (g ~ 1e-7).
__device__ __forceinline__ float inv_norm2_m1(float2 w) {
    const float p1 = w.x * w.x, p2 = w.y * w.y;
    const float e1 = fmaf(w.x, w.x, -p1), e2 = fmaf(w.y, w.y, -p2);
    const float big = fmaxf(p1, p2), small = fminf(p1, p2);
    const float g0 = (big >= 0.5f) ? (big - 1.0f) + small : (p1 - 0.5f) + (p2 - 0.5f);
    const float g = g0 + (e1 + e2);
    return fmaf(g, g, -g);
}

__device__ __forceinline__ int bitrev(int x, int bits) {
    return bits == 0 ? 0 : (int)(__brev((unsigned)x) >> (32 - bits));
}

}  // namespace ofx
