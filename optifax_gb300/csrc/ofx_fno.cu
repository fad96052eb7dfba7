// ofx_fno.cu -- Fourier-neural-operator surrogate of one crystal pass: forward,
// backward and AdamW on the GPU.  No reference counterpart (the reference has no
// learned component).
//
// Network (fixed sizes): input x[b][6][L] (4 field channels, one constant
// conditioning channel and the bin coordinate over L frequency bins), lifting to
// width 64, four Fourier
// layers h <- act(SpecConv(h) + Wp h + bias) with 32 retained modes (no activation
// after the last), projection to 4 channels plus a residual connection to the
// first 4 input channels: y = x[:4] + Q h + q.
//
// A layer's two products with a spatial output -- inverse transform and pointwise mix
// forward, their transposes backward -- run in one kernel per 128 bins (k_layer), whose
// epilogue adds them, applies bias and GELU (or its derivative) and writes what the next
// products read; no FP32 intermediate goes through memory but the kept pre-activation.
//
// Data layouts (per batch of B samples): "channel-major" Hc[c][b][x] and
// "point-major" Ht[b][x][c] copies of every activation, so that every product is
// an A . B^T GEMM with both operands K-major for the tensor-core kernel
// (optifax_gemm_bf16):
//   spectral transform   S[(c,b)][m'] = Hc . F^T         (F: 64 x L, m' = 2m + re/im)
//   inverse transform    Y1[x][o] = G . T_b^T            (G: L x 64, T: [b][o][m'])
//   pointwise mix        Y2[x][o] = Ht_b . Wp^T          (Wp: 64 x 64, [o][c])
//   weight gradient      dWp[o][c]    = dZc[o][(b,x)] . Hc[c][(b,x)]^T
//   backward transforms  dT = dZc . GT^T, dH = FT . dS_b^T + dZt_b . WpT^T
// The per-mode complex channel mixing T[b][o][m] = sum_c S[(c,b)][m] W[c][o][m]
// and the element-wise parts run on the CUDA cores.  GEMM operands and
// activations are BF16; accumulation, pre-activations, gradients, biases, the
// master weights and the Adam moments are FP32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../include/optifax.h"
#include "ofx_fft.cuh"
#include "ofx_tc.cuh"
#include "ofx_tmap.cuh"

typedef __nv_bfloat16 bf16;

using ofx_tc::dep_launch;
using ofx_tc::dep_wait;
using ofx_tc::launch_dep;

namespace {

constexpr int W = 64, MODES = 32, NLAYER = 4, CIN = 6, COUT = 4, SPEC = 2 * MODES;
constexpr long long LAYER_WS = (long long)W * W * MODES * 2;   // [c][o][m][re,im]
constexpr long long LAYER_SIZE = LAYER_WS + W * W + W;         // Ws, Wp [o][c], bias [o]
constexpr long long OFF_P = 0;                                 // [W][CIN]
constexpr long long OFF_PB = OFF_P + W * CIN;                  // [W]
constexpr long long OFF_L0 = OFF_PB + W;
constexpr long long OFF_Q = OFF_L0 + NLAYER * LAYER_SIZE;      // [COUT][W]
constexpr long long OFF_QB = OFF_Q + COUT * W;                 // [COUT]
constexpr long long N_PARAMS = OFF_QB + COUT;
constexpr long long off_ws(int l) { return OFF_L0 + l * LAYER_SIZE; }
constexpr long long off_wp(int l) { return off_ws(l) + LAYER_WS; }
constexpr long long off_b(int l) { return off_wp(l) + W * W; }
static_assert(off_wp(0) % 8 == 0 && LAYER_SIZE % 8 == 0, "BF16 GEMM operands must stay 16-byte aligned");

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float z) {
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// ---- tables --------------------------------------------------------------
__global__ void k_dft_tables(int L, bf16* F, bf16* FT, bf16* G, bf16* GT) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)SPEC * L) return;
    const int mp = (int)(i / L), x = (int)(i % L), m = mp >> 1;
    const long long ph = ((long long)m * x) % L;
    float s, c;
    sincospif(2.f * (float)ph / (float)L, &s, &c);
    const float f = (mp & 1) ? -s : c;
    const float g = f * (m == 0 ? 1.f : 2.f) / (float)L;
    F[(long long)mp * L + x] = __float2bfloat16(f);
    FT[(long long)x * SPEC + mp] = __float2bfloat16(f);
    G[(long long)x * SPEC + mp] = __float2bfloat16(g);
    GT[(long long)mp * L + x] = __float2bfloat16(g);
}

__global__ void k_refresh(const float* __restrict__ master, bf16* wb, bf16* wpt) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < N_PARAMS) wb[i] = __float2bfloat16(master[i]);
    if (i < (long long)NLAYER * W * W) {
        const int l = (int)(i / (W * W)), r = (int)(i % (W * W)), c = r / W, o = r % W;
        wpt[i] = __float2bfloat16(master[off_wp(l) + (long long)o * W + c]);
    }
}

// ---- forward -------------------------------------------------------------
// A thread takes one bin and 16 channels; a warp 32 bins of one channel group
__global__ void __launch_bounds__(256) k_lift(const float* __restrict__ x, const bf16* __restrict__ Pw,
                                              const float* __restrict__ pb, int B, int L, bf16* __restrict__ Hc,
                                              bf16* __restrict__ Ht) {
    __shared__ float sP[W * CIN];
    __shared__ float sb[W];
    dep_launch();
    dep_wait();
    for (int i = threadIdx.x; i < W * CIN; i += 256) sP[i] = __bfloat162float(Pw[i]);
    for (int i = threadIdx.x; i < W; i += 256) sb[i] = pb[i];
    __syncthreads();
    const int c0 = (threadIdx.x >> 6) * 16;
    const long long idx = blockIdx.x * 64LL + (threadIdx.x & 63);
    if (idx >= (long long)B * L) return;
    const int b = (int)(idx / L), xx = (int)(idx % L);
    float in[CIN];
#pragma unroll
    for (int i = 0; i < CIN; ++i) in[i] = x[((long long)b * CIN + i) * L + xx];
    uint4 pack[2];
    bf16* hp = reinterpret_cast<bf16*>(pack);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int c = c0 + j;
        float h = sb[c];
#pragma unroll
        for (int i = 0; i < CIN; ++i) h = fmaf(sP[c * CIN + i], in[i], h);
        hp[j] = __float2bfloat16(h);
        Hc[((long long)c * B + b) * L + xx] = hp[j];
    }
    uint4* dst = reinterpret_cast<uint4*>(Ht + idx * W + c0);
    dst[0] = pack[0];
    dst[1] = pack[1];
}

// Channel mixing per mode: out[b][u][m] = sum_v in[(v,b)][m] w (or conj w) with w =
// Ws[v][u][m] (forward, u = o) or Ws[u][v][m] conjugated (backward, u = c).  The sum is
// rounded to BF16 for a whole row of the next product, so its order is part of the result:
// one FP32 accumulator pair per output, v = 0..63 in turn (in eight partial sums a last
// bit before the rounding moved elements of small batches' gradients by up to 1e-3).
// What cost time in that order were its loads, one dependent step after the other, so a
// block of U outputs and MB samples first copies its rows of `in` and its weights to shared
// memory, all copies in flight at once; then a warp per (output, sample), lane = mode,
// runs the 64 steps (32 samples: 6.8 us cold, 14 in eight partial sums from global memory).
template <int U, int MB>
struct Mix {
    static constexpr int IN = W * MB * SPEC;                              // floats: [v][sample][2 m]
    static constexpr size_t smem = sizeof(float) * IN + sizeof(__nv_bfloat162) * W * U * MODES;
};
template <bool BWD, int U, int MB>
__global__ void __launch_bounds__(256) k_mix(const float* __restrict__ in, const bf16* __restrict__ Ws, int B,
                                             bf16* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* s_in = reinterpret_cast<float*>(smem_raw);
    __nv_bfloat162* s_w = reinterpret_cast<__nv_bfloat162*>(s_in + Mix<U, MB>::IN);      // [v][output][mode]
    const int u0 = blockIdx.x * U, b0 = blockIdx.y * MB, n = min(MB, B - b0);
    dep_launch();
    dep_wait();
    for (int i = threadIdx.x; i < W * MB * (SPEC / 4); i += 256) {
        const int row = i / (SPEC / 4), c4 = 4 * (i % (SPEC / 4)), v = row / MB, k = row % MB;
        if (k < n) ofx_tc::cp_async16(s_in + row * SPEC + c4, in + ((long long)v * B + b0 + k) * SPEC + c4);
    }
    for (int i = threadIdx.x; i < W * U * (MODES / 4); i += 256) {
        const int row = i / (MODES / 4), m4 = 4 * (i % (MODES / 4)), v = row / U, q = row % U;
        const long long wi = BWD ? ((long long)(u0 + q) * W + v) : ((long long)v * W + u0 + q);
        ofx_tc::cp_async16(s_w + row * MODES + m4, Ws + (wi * MODES + m4) * 2);
    }
    ofx_tc::cp_async_wait();
    __syncthreads();
    const int m = threadIdx.x & 31, q = (threadIdx.x >> 5) % U, k = (threadIdx.x >> 5) / U;
    if (k >= n) return;
    float ar = 0.f, ai = 0.f;
#pragma unroll 8
    for (int v = 0; v < W; ++v) {
        const float2 s = *reinterpret_cast<const float2*>(s_in + (v * MB + k) * SPEC + 2 * m);
        const __nv_bfloat162 w = s_w[(v * U + q) * MODES + m];
        const float wr = __low2float(w), wi = __high2float(w);
        if (BWD) {
            ar = fmaf(s.x, wr, fmaf(s.y, wi, ar));
            ai = fmaf(s.y, wr, fmaf(-s.x, wi, ai));
        } else {
            ar = fmaf(s.x, wr, fmaf(-s.y, wi, ar));
            ai = fmaf(s.x, wi, fmaf(s.y, wr, ai));
        }
    }
    *reinterpret_cast<__nv_bfloat162*>(out + ((long long)(b0 + k) * W + u0 + q) * SPEC + 2 * m) =
        __floats2bfloat162_rn(ar, ai);
}
// One output and one sample per block up to 8 samples (64 blocks a sample, 24 KB each);
// above, where the blocks fill the GPU and reading `in` once per output is what costs, four
// outputs and two samples (64 KB, so a third of the reads)
constexpr int MIXU = 4, MIXB = 2;
template <bool BWD>
void launch_mix(const float* in, const bf16* Ws, int B, bf16* out, cudaStream_t st) {
    if (B <= 8)
        launch_dep(k_mix<BWD, 1, 1>, dim3(W, B), dim3(256), Mix<1, 1>::smem, st, in, Ws, B, out);
    else
        launch_dep(k_mix<BWD, MIXU, MIXB>, dim3(W / MIXU, (B + MIXB - 1) / MIXB), dim3(256), Mix<MIXU, MIXB>::smem, st,
                   in, Ws, B, out);
}

// ---- one layer's spatial part ---------------------------------------------
// A CTA takes 128 bins of one sample: D1[x][u] = R . X_b^T (R: G or FT, X: T or dS) and
// D2[x][u] = H_b . V^T (H: Ht or dZt, V: Wp or its transpose), K = 64 each, two
// tcgen05 accumulators of 64 columns; thread = bin in the epilogue.  48 KB of operands
// and 128 TMEM columns, so four CTAs share an SM and their loads, products and epilogues
// overlap.  Bound by the epilogue's traffic (batch 32, 4096 bins: 84 MB forward).
enum { LAYER_FWD = 0, LAYER_BWD = 1, LAYER_BWD_IN = 2 };
struct LayerArgs {
    const float* bias;      // FWD
    float* Z;               // FWD: pre-activation out [c][b][x] (or null); BWD: in
    bf16 *Hc, *Ht;          // FWD: activation; BWD: dZ
    const float* x;         // BWD_IN: network input [b][CIN][x]
    float* db;              // BWD: bias gradient; BWD_IN: this launch's partial sums [CTA][W][8]
    int* err;
    int B, L, act;
};
constexpr int LA = 128 * 64 * 2, LB = 64 * 64 * 2;
constexpr int LAYER_SMEM = 2 * LA + 2 * LB + 1024;

template <int MODE>
__global__ void __launch_bounds__(128, 4)
    k_layer(const __grid_constant__ CUtensorMap tmR, const __grid_constant__ CUtensorMap tmH,
            const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmV, LayerArgs a) {
    using namespace ofx_tc;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full, accum;
    __shared__ uint32_t tmem_slot;
    __shared__ float s_bias[W];
    const int warp = threadIdx.x >> 5;
    const int b = blockIdx.y, x0 = blockIdx.x * 128;
    if (threadIdx.x == 0) {
        mbar_init(&full, 1);
        mbar_init(&accum, 1);
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 128);
    __syncthreads();   // the next grid may take tensor memory only once this CTA has its own
    dep_launch();
    dep_wait();
    if (MODE == LAYER_FWD && threadIdx.x < W) s_bias[threadIdx.x] = a.bias[threadIdx.x];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (threadIdx.x == 0) {
        mbar_expect_tx(&full, 2 * LA + 2 * LB);
        tma_load_2d(tiles, &tmR, 0, x0, &full);
        tma_load_2d(tiles + LA, &tmH, 0, b * a.L + x0, &full);
        tma_load_2d(tiles + 2 * LA, &tmX, 0, b * W, &full);
        tma_load_2d(tiles + 2 * LA + LB, &tmV, 0, 0, &full);
        if (mbar_wait(&full, 0)) {
            tc_fence_after();
            constexpr uint32_t idesc = idesc_bf16_f32(128, 64);
#pragma unroll
            for (int d = 0; d < 2; ++d)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mma_bf16(tmem + 64 * d, desc_kmajor_sw128(smem_u32(tiles + d * LA) + kk * 32),
                             desc_kmajor_sw128(smem_u32(tiles + 2 * LA + d * LB) + kk * 32), idesc, kk > 0 ? 1u : 0u);
        }
        mma_commit(&accum);
    }
    __syncwarp();
    // a load that did not arrive in time leaves `full` in its first phase: every thread sees it
    const bool ok = mbar_wait(&accum, 0) && mbar_try_wait(&full, 0);
    __syncwarp();
    tc_fence_after();

    const int x = x0 + threadIdx.x;
    const bool live = ok && x < a.L;
    const uint32_t taddr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    float* gt = reinterpret_cast<float*>(tiles);              // BWD: g as [x][u], padded (operands are consumed)
    constexpr int LDG = W + 1;
    if (MODE != LAYER_FWD) __syncthreads();
#pragma unroll 1
    for (int u0 = 0; u0 < W; u0 += 16) {
        float d1[16], d2[16];
        tmem_ld16(taddr + u0, d1);
        tmem_ld16(taddr + 64 + u0, d2);
        uint4 pack[2];
        bf16* hp = reinterpret_cast<bf16*>(pack);
        if (MODE == LAYER_FWD) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float z = d1[j] + d2[j] + s_bias[u0 + j];
                const long long o = ((long long)(u0 + j) * a.B + b) * a.L + x;
                if (a.Z && live) a.Z[o] = z;
                hp[j] = __float2bfloat16(a.act ? gelu(z) : z);
                if (live) a.Hc[o] = hp[j];
            }
        } else {
            float zv[16];                                     // every load in flight before any store
            if (MODE == LAYER_BWD) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    zv[j] = live ? a.Z[((long long)(u0 + j) * a.B + b) * a.L + x] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float g = d1[j] + d2[j];
                if (MODE == LAYER_BWD) {
                    g *= gelu_d(zv[j]);
                    hp[j] = __float2bfloat16(g);
                    if (live) a.Hc[((long long)(u0 + j) * a.B + b) * a.L + x] = hp[j];
                }
                gt[threadIdx.x * LDG + u0 + j] = live ? g : 0.f;
            }
        }
        if (MODE != LAYER_BWD_IN && live) {
            uint4* dst = reinterpret_cast<uint4*>(a.Ht + ((long long)b * a.L + x) * W + u0);
            dst[0] = pack[0];
            dst[1] = pack[1];
        }
    }
    if (MODE == LAYER_BWD) {
        __syncthreads();
        const int c = threadIdx.x & 63, h = threadIdx.x >> 6;
        float s = 0.f;
#pragma unroll 8
        for (int r = 0; r < 64; ++r) s += gt[(h * 64 + r) * LDG + c];
        __syncthreads();
        if (h) gt[c] = s;
        __syncthreads();
        if (!h) atomicAdd(&a.db[c], s + gt[c]);
    }
    if (MODE == LAYER_BWD_IN) {
        // dP[c][i] = sum_x g[x][c] x_i, dp[c] = sum_x g[x][c]
        float* xs = gt + 128 * LDG;                           // [x][8]: the inputs and a one
        for (int i = 0; i < 8; ++i)
            xs[threadIdx.x * 8 + i] =
                i < CIN ? (live ? a.x[((long long)b * CIN + i) * a.L + x] : 0.f) : (i == CIN ? 1.f : 0.f);
        __syncthreads();
        const int c = threadIdx.x & 63, h = threadIdx.x >> 6;
        float s[CIN + 1] = {};
#pragma unroll 4
        for (int r = 0; r < 64; ++r) {
            const float g = gt[(h * 64 + r) * LDG + c];
            const float4 p = *reinterpret_cast<const float4*>(xs + (h * 64 + r) * 8);
            const float4 q = *reinterpret_cast<const float4*>(xs + (h * 64 + r) * 8 + 4);
            s[0] = fmaf(g, p.x, s[0]); s[1] = fmaf(g, p.y, s[1]); s[2] = fmaf(g, p.z, s[2]); s[3] = fmaf(g, p.w, s[3]);
            s[4] = fmaf(g, q.x, s[4]); s[5] = fmaf(g, q.y, s[5]); s[6] += g;
        }
        __syncthreads();
        if (h)
            for (int i = 0; i <= CIN; ++i) gt[c * 8 + i] = s[i];
        __syncthreads();
        // partial sums to memory, one row per CTA: 448 atomics from each of 1024 CTAs queued on
        // the same few sectors for 50 us
        if (!h) {
            float4* row = reinterpret_cast<float4*>(a.db + ((long long)b * gridDim.x + blockIdx.x) * W * 8 + c * 8);
            row[0] = make_float4(s[0] + gt[c * 8], s[1] + gt[c * 8 + 1], s[2] + gt[c * 8 + 2], s[3] + gt[c * 8 + 3]);
            row[1] = make_float4(s[4] + gt[c * 8 + 4], s[5] + gt[c * 8 + 5], s[6] + gt[c * 8 + 6], 0.f);
        }
    }
    if (!ok && threadIdx.x == 0) {
        atomicOr(a.err, 1);
        mbar_wait(&full, 0);               // copies still in flight land before the memory is released
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

// y[b][j][x] = x[b][j][x] + (q[j] + sum_c Q[j][c] h[b][x][c]), c in turn: the loss's
// gradient is a difference of y that is rounded to BF16.  Four lanes share a bin, one output
// each; they read the same 16 bytes of its row, and of the weights 16 bytes each, four banks
// apart (32 samples of 4096 bins: 14.0 us cold, waiting on its loads; 10.5 with 16 channels a
// lane, whose sums had another order).
__global__ void __launch_bounds__(256) k_proj_fwd(const bf16* __restrict__ Ht, const bf16* __restrict__ Qw,
                                                  const float* __restrict__ qb, const float* __restrict__ xin, int B,
                                                  int L, float* __restrict__ y) {
    constexpr int LDQ = W + 4;
    __shared__ __align__(16) float sQ[COUT * LDQ];
    dep_launch();
    dep_wait();
    if (threadIdx.x < COUT * W) sQ[threadIdx.x / W * LDQ + threadIdx.x % W] = __bfloat162float(Qw[threadIdx.x]);
    __syncthreads();
    const long long idx = blockIdx.x * 64LL + (threadIdx.x >> 2);
    const int j = threadIdx.x & 3;
    if (idx >= (long long)B * L) return;
    const uint4* src = reinterpret_cast<const uint4*>(Ht + idx * W);
    uint4 u[W / 8];
#pragma unroll
    for (int i = 0; i < W / 8; ++i) u[i] = src[i];
    float acc = qb[j];
#pragma unroll
    for (int c = 0; c < W; c += 4) {
        const float4 q = *reinterpret_cast<const float4*>(sQ + j * LDQ + c);
        const bf16* hp = reinterpret_cast<const bf16*>(&u[c / 8]) + c % 8;
        acc = fmaf(q.x, __bfloat162float(hp[0]), acc);
        acc = fmaf(q.y, __bfloat162float(hp[1]), acc);
        acc = fmaf(q.z, __bfloat162float(hp[2]), acc);
        acc = fmaf(q.w, __bfloat162float(hp[3]), acc);
    }
    const int b = (int)(idx / L), xx = (int)(idx % L);
    y[((long long)b * COUT + j) * L + xx] = xin[((long long)b * CIN + j) * L + xx] + acc;
}

// dP[c][i] and dp[c] from k_layer's partial rows [n][W][8]; block: 32 of the 512 columns,
// 8 row lanes; blockIdx.y splits the rows
__global__ void __launch_bounds__(256) k_lift_sum(const float* __restrict__ part, int n, float* __restrict__ dP,
                                                  float* __restrict__ dp) {
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, col = blockIdx.x * 32 + lane;
    float s = 0.f;
    dep_launch();
    dep_wait();
#pragma unroll 4
    for (int r = blockIdx.y * 8 + wp; r < n; r += 8 * gridDim.y) s += part[(long long)r * (W * 8) + col];
    red[wp][lane] = s;
    __syncthreads();
    if (wp == 0) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += red[i][lane];
        const int c = col >> 3, i = col & 7;
        if (i < CIN) atomicAdd(&dP[c * CIN + i], t);
        else if (i == CIN) atomicAdd(&dp[c], t);
    }
}

// ---- loss and backward ---------------------------------------------------
// loss = sum_i w_(sample of i) (y_i - t_i)^2 / n  (w = 1 without sample weights)
__global__ void k_loss(const float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ w,
                       long long per_sample, long long n, float inv_n, float* __restrict__ dy,
                       float* __restrict__ loss) {
    __shared__ float red[32];
    float part = 0.f;
    dep_launch();
    dep_wait();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float d = y[i] - t[i];
        const float wi = w ? w[i / per_sample] : 1.f;
        dy[i] = 2.f * d * inv_n * wi;
        part = fmaf(wi * d, d, part);
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) atomicAdd(loss, v * inv_n);
    }
}

// dH4 = Q^T dy (the last layer has no activation, so this is dZ of layer 3) -> dZc, dZt;
// dQ[j][c] = sum_(b,x) dy[b][j][x] h[b][x][c], dq[j] = sum dy[b][j][x]; the bias gradient
// is Q^T dq.  A block takes 256 bins of one sample: a thread per bin for dZ, then a lane
// per channel pair and a warp per 32 bins for the sums.
__global__ void __launch_bounds__(256) k_proj_bwd(const float* __restrict__ dy, const bf16* __restrict__ Qw,
                                                  const bf16* __restrict__ Ht, int B, int L, bf16* __restrict__ dZc,
                                                  bf16* __restrict__ dZt, float* __restrict__ db,
                                                  float* __restrict__ dQ, float* __restrict__ dq) {
    __shared__ float sQ[COUT * W];
    __shared__ float4 sd[256];
    __shared__ float red[8][COUT * W];
    __shared__ float rq[8][COUT];
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, b = blockIdx.y, x = blockIdx.x * 256 + t;
    dep_launch();
    dep_wait();
    for (int i = t; i < COUT * W; i += 256) sQ[i] = __bfloat162float(Qw[i]);
    const bool live = x < L;
    float d[COUT] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
#pragma unroll
        for (int j = 0; j < COUT; ++j) d[j] = dy[((long long)b * COUT + j) * L + x];
    }
    sd[t] = make_float4(d[0], d[1], d[2], d[3]);
    __syncthreads();
    if (live) {
        uint4* dst = reinterpret_cast<uint4*>(dZt + ((long long)b * L + x) * W);
#pragma unroll
        for (int c0 = 0; c0 < W; c0 += 8) {
            uint4 pack;
            bf16* gp = reinterpret_cast<bf16*>(&pack);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float g = 0.f;
#pragma unroll
                for (int j = 0; j < COUT; ++j) g = fmaf(sQ[j * W + c0 + i], d[j], g);
                gp[i] = __float2bfloat16(g);
                dZc[((long long)(c0 + i) * B + b) * L + x] = gp[i];
            }
            dst[c0 / 8] = pack;
        }
    }
    // a lane's channels 2 lane, 2 lane + 1 over the warp's 32 bins
    float acc[2 * COUT] = {};
    const int xw = blockIdx.x * 256 + wp * 32, rows = min(32, L - xw);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(Ht + ((long long)b * L + xw) * W) + lane;
#pragma unroll 8
    for (int r = 0; r < rows; ++r) {
        const __nv_bfloat162 v = h[r * (W / 2)];
        const float h0 = __low2float(v), h1 = __high2float(v);
        const float4 e = sd[wp * 32 + r];
        acc[0] = fmaf(e.x, h0, acc[0]); acc[1] = fmaf(e.x, h1, acc[1]);
        acc[2] = fmaf(e.y, h0, acc[2]); acc[3] = fmaf(e.y, h1, acc[3]);
        acc[4] = fmaf(e.z, h0, acc[4]); acc[5] = fmaf(e.z, h1, acc[5]);
        acc[6] = fmaf(e.w, h0, acc[6]); acc[7] = fmaf(e.w, h1, acc[7]);
    }
#pragma unroll
    for (int j = 0; j < COUT; ++j) {
        red[wp][j * W + 2 * lane] = acc[2 * j];
        red[wp][j * W + 2 * lane + 1] = acc[2 * j + 1];
        float s = d[j];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) rq[wp][j] = s;
    }
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[i][t];
    atomicAdd(&dQ[t], s);
    if (t < W) {
        float g = 0.f;
        for (int j = 0; j < COUT; ++j) {
            float q = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) q += rq[i][j];
            g = fmaf(sQ[j * W + t], q, g);
            if (t == 0) atomicAdd(&dq[j], q);
        }
        atomicAdd(&db[t], g);
    }
}

// dW[c][o][m] = sum_b conj(S[(c,b)][m]) dT[(o,b)][m]
__global__ void k_mix_bwd_dw(const float* __restrict__ dT, const float* __restrict__ S, int B, float* __restrict__ dW) {
    dep_launch();
    dep_wait();
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)W * W * MODES) return;
    const int m = (int)(idx % MODES);
    const long long t = idx / MODES;
    const int o = (int)(t % W), c = (int)(t / W);
    float ar = 0.f, ai = 0.f;
    for (int b = 0; b < B; ++b) {
        const float* s = S + ((long long)c * B + b) * SPEC + 2 * m;
        const float* d = dT + ((long long)o * B + b) * SPEC + 2 * m;
        ar = fmaf(s[0], d[0], fmaf(s[1], d[1], ar));
        ai = fmaf(s[0], d[1], fmaf(-s[1], d[0], ai));
    }
    dW[(((long long)c * W + o) * MODES + m) * 2] = ar;
    dW[(((long long)c * W + o) * MODES + m) * 2 + 1] = ai;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * ((mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * p[i]);
}

// ---- OPO fast-forward: spectra <-> network channels ------------------------
// The crop is n_bins consecutive bins of an N-point spectrum (natural FFT order)
// starting at bin k0 (wrapping at N); bins j < split form the signal band.
__global__ void k_ff_encode(const float2* __restrict__ Y, long long ystride, int N, int k0, int L, int split,
                            float pump_scale, const float* __restrict__ sigma_in, float* __restrict__ x, int nch,
                            float* __restrict__ sigma_out) {
    __shared__ float red[32];
    __shared__ float s_sigma;
    const int p = blockIdx.x;
    const float2* y = Y + p * ystride;
    if (sigma_in) {
        if (threadIdx.x == 0) s_sigma = sigma_in[p];
    } else {
        float acc = 0.f;
        for (int j = threadIdx.x; j < split; j += blockDim.x) {
            const float2 v = y[(k0 + j) % N];
            acc = fmaf(v.x, v.x, fmaf(v.y, v.y, acc));
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            float tot = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
            float sg = sqrtf(tot / (float)(split > 0 ? split : 1));
            const float floor_ = 1e-30f * pump_scale;
            if (!(sg > floor_)) sg = floor_;
            s_sigma = sg;
            if (sigma_out) sigma_out[p] = sg;
        }
    }
    __syncthreads();
    const float sg = s_sigma, inv_s = 1.f / sg, inv_p = 1.f / pump_scale;
    const float lg = log10f(sg * inv_p);
    float* xo = x + (long long)p * nch * L;
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const float2 v = y[(k0 + j) % N];
        const bool sb = j < split;
        xo[j] = sb ? 0.f : v.x * inv_p;
        xo[L + j] = sb ? 0.f : v.y * inv_p;
        xo[2 * L + j] = sb ? v.x * inv_s : 0.f;
        xo[3 * L + j] = sb ? v.y * inv_s : 0.f;
        if (nch > 4) {
            xo[4 * L + j] = lg;
            xo[5 * L + j] = (float)j / (float)L;
        }
    }
}

// X = (decoded network output or X_in) times lin; Y_next = X fb + pump; energy += sum tally_w |X|^2
__global__ void k_ff_step(const float* __restrict__ y, const float* __restrict__ sigma, const float2* __restrict__ X_in,
                          const float2* __restrict__ fb, const float2* __restrict__ pump,
                          const float2* __restrict__ lin, const float* __restrict__ tw, int N, int k0, int L,
                          int split, float pump_scale, float2* __restrict__ X_out, float2* __restrict__ Y_next,
                          double* __restrict__ energy) {
    __shared__ double red[32];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0;
    dep_launch();
    dep_wait();
    if (k < N) {
        float2 X = make_float2(0.f, 0.f);
        if (y) {
            const int j = (k - k0 + N) % N;
            if (j < L) {
                if (j < split) {
                    const float sg = sigma[0];
                    X = make_float2(y[2 * L + j] * sg, y[3 * L + j] * sg);
                } else {
                    X = make_float2(y[j] * pump_scale, y[L + j] * pump_scale);
                }
            }
        } else {
            X = X_in[k];
        }
        if (lin) {
            const float2 d = lin[k];
            X = make_float2(X.x * d.x - X.y * d.y, X.x * d.y + X.y * d.x);
        }
        if (X_out) X_out[k] = X;
        const float2 f = fb[k], pp = pump[k];
        Y_next[k] = make_float2(X.x * f.x - X.y * f.y + pp.x, X.x * f.y + X.y * f.x + pp.y);
        if (tw) e = (double)tw[k] * ((double)X.x * X.x + (double)X.y * X.y);
    }
    if (energy) {
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
            atomicAdd(energy, tot);
        }
    }
}

// ---- OPO fast-forward, envelope representation ---------------------------
// A band is the set of bins whose signed offset o from the band's carrier bin kc
// (natural FFT order of the N-point spectrum) lies in [lo, hi), |o| < L/2.  Its
// envelope is e_j = sum_o b_o exp(+2 pi i o j / L), j < L: the band demodulated to
// its carrier and sampled L times over the window.
struct EnvBand {
    int kc, lo, hi;
};

__device__ __forceinline__ int env_bin(const EnvBand& b, int N, int L, int j, bool* in) {
    const int o = j < L / 2 ? j : j - L;
    *in = o >= b.lo && o < b.hi;
    int k = (b.kc + o) % N;
    return k < 0 ? k + N : k;
}

constexpr int ENV_MAX = 4096, ENV_T = 512;

// Slot of point m: the strided passes and the last pass's bit-reversed scatter spread
// over the banks
__device__ __forceinline__ int env_slot(int m) { return m ^ ((m >> 4) & 15); }

// Quarter period of exp(-2 pi i m / L)
__device__ __forceinline__ void env_table(float2* quad, int L) {
    for (int i = threadIdx.x; i < (L + 3) / 4; i += ENV_T) {
        float sn, cs;
        sincospif(-2.f * (float)i / (float)L, &sn, &cs);
        quad[i] = make_float2(cs, sn);
    }
}
__device__ __forceinline__ float2 env_tw(const float2* quad, int logL, int m) {
    if (logL < 2) return make_float2(1.f, 0.f);              // L = 2 has the factor 1 only
    const float2 w = quad[m & ((1 << (logL - 2)) - 1)];
    const int k = m >> (logL - 2);                           // times (-i)^k
    const float2 u = (k & 1) ? make_float2(w.y, -w.x) : w;
    return (k & 2) ? make_float2(-u.x, -u.y) : u;
}

// One decimation-in-frequency pass of radix R over blocks of 2^logB points; the last
// pass leaves frequency k in slot k.
template <int R>
__device__ void env_pass(float2* sm, const float2* quad, int logL, int logB) {
    const int L = 1 << logL, LR = (1 << logB) / R, b = threadIdx.x;   // L / R <= ENV_T
    const bool live = b < L / R, last = LR == 1;
    const int off = b & (LR - 1), base = (b - off) * R + off;
    float2 v[R];
    if (live) {
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = sm[env_slot(base + q * LR)];
        ofx::dftp<R>(v);
    }
    if (last) __syncthreads();
    if (live) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = ofx::brev4(q, ofx::ilog2(R));
            if (last) sm[env_slot(__brev((unsigned)(base + q)) >> (32 - logL))] = v[q];
            else sm[env_slot(base + q * LR)] = q ? ofx::cmul(v[q], env_tw(quad, logL, (off * r) << (logL - logB))) : v[q];
        }
    }
    __syncthreads();
}

// exp(-2 pi i j k / L) transform of the 2^logL points at env_slot(j), in place and in
// natural order, by ENV_T threads.  Radix 8 with one shared-memory table: the previous
// radix-2 form called sincospi in each of the L/2 log2(L) butterflies (25 us at 4096).
__device__ void env_fft(float2* sm, const float2* quad, int logL) {
    __syncthreads();
    int logB = logL;
    for (; logB >= 3; logB -= 3) env_pass<8>(sm, quad, logL, logB);
    if (logB == 2) env_pass<4>(sm, quad, logL, logB);
    if (logB == 1) env_pass<2>(sm, quad, logL, logB);
}

// grid (spectra, 2 bands): envelopes -> channels 0/1 (pump / pump_scale), 2/3
// (signal / sigma), 4 log10(sigma / pump_scale), 5 j / L
__global__ void __launch_bounds__(ENV_T) k_ff_encode_env(const float2* __restrict__ Y, long long ystride, int N, int L, int logL, EnvBand bp,
                                EnvBand bs, float pump_scale, const float* __restrict__ sigma_in,
                                float* __restrict__ x, int nch, float* __restrict__ sigma_out) {
    __shared__ float2 sm[ENV_MAX];
    __shared__ float2 quad[ENV_MAX / 4];
    __shared__ float red[32];
    __shared__ float s_sig;
    const int p = blockIdx.x, band = blockIdx.y;
    const EnvBand bd = band ? bs : bp;
    const float2* y = Y + p * ystride;
    dep_launch();
    env_table(quad, L);
    dep_wait();
    // exp(+...): real and imaginary parts exchanged before and after
    for (int j = threadIdx.x; j < L; j += ENV_T) {
        bool in;
        const int k = env_bin(bd, N, L, j, &in);
        const float2 u = in ? y[k] : make_float2(0.f, 0.f);
        sm[env_slot(j)] = make_float2(u.y, u.x);
    }
    env_fft(sm, quad, logL);
    float scale = 1.f / pump_scale, sg = 1.f;
    if (band == 1) {
        if (sigma_in) {
            if (threadIdx.x == 0) s_sig = sigma_in[p];
        } else {
            float acc = 0.f;
            for (int j = threadIdx.x; j < L; j += ENV_T) acc = fmaf(sm[j].x, sm[j].x, fmaf(sm[j].y, sm[j].y, acc));
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
            __syncthreads();
            if (threadIdx.x == 0) {
                float tot = 0.f;
                for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
                float v = sqrtf(tot / (float)L);
                const float floor_ = 1e-30f * pump_scale;
                if (!(v > floor_)) v = floor_;
                s_sig = v;
                if (sigma_out) sigma_out[p] = v;
            }
        }
        __syncthreads();
        sg = s_sig;
        scale = 1.f / sg;
    }
    float* xo = x + (long long)p * nch * L;
    const float lg = log10f(sg / pump_scale);
    for (int j = threadIdx.x; j < L; j += ENV_T) {
        const float2 u = sm[env_slot(j)];
        xo[(2 * band) * L + j] = u.y * scale;
        xo[(2 * band + 1) * L + j] = u.x * scale;
        if (band == 1 && nch > 4) {
            xo[4 * L + j] = lg;
            xo[5 * L + j] = (float)j / (float)L;
        }
    }
}

// Blocks 0 and 1: network output envelopes -> the band bins of X; the others clear the
// bins outside both bands, ENV_T each
__global__ void __launch_bounds__(ENV_T)
    k_ff_decode_env(const float* __restrict__ y, const float* __restrict__ sigma, int N, int L, int logL, EnvBand bp,
                    EnvBand bs, float pump_scale, float2* __restrict__ X) {
    __shared__ float2 sm[ENV_MAX];
    __shared__ float2 quad[ENV_MAX / 4];
    dep_launch();
    if (blockIdx.x >= 2) {
        dep_wait();
        const int k = (blockIdx.x - 2) * ENV_T + threadIdx.x;
        bool in = k >= N;
        for (const EnvBand& b : {bp, bs}) {
            int o = k - b.kc;
            if (o < 0) o += N;
            if (o >= N - L / 2) o -= N;
            in = in || (o >= b.lo && o < b.hi);
        }
        if (!in) X[k] = make_float2(0.f, 0.f);
        return;
    }
    const int band = blockIdx.x;
    const EnvBand bd = band ? bs : bp;
    env_table(quad, L);
    dep_wait();
    for (int j = threadIdx.x; j < L; j += ENV_T)
        sm[env_slot(j)] = make_float2(y[(2 * band) * L + j], y[(2 * band + 1) * L + j]);
    env_fft(sm, quad, logL);
    const float scale = (band ? sigma[0] : pump_scale) / (float)L;
    for (int j = threadIdx.x; j < L; j += ENV_T) {
        bool in;
        const int k = env_bin(bd, N, L, j, &in);
        const float2 u = sm[env_slot(j)];
        if (in) X[k] = make_float2(u.x * scale, u.y * scale);
    }
}

inline unsigned nblk(long long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

struct optifax_fno_s {
    int device = 0, L = 0, maxB = 0;
    float *master = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    bf16 *wb = nullptr, *wpt = nullptr;
    bf16 *F = nullptr, *FT = nullptr, *G = nullptr, *GT = nullptr;
    bf16 *Hc[NLAYER + 1] = {}, *Ht[NLAYER + 1] = {};
    float* Z[NLAYER - 1] = {};
    float *S[NLAYER] = {}, *dT[NLAYER] = {};    // one allocation each, batch rows [layer][64 B][64]
    bf16 *T = nullptr, *dS = nullptr, *dZc = nullptr, *dZt = nullptr;
    float *y = nullptr, *dy = nullptr, *loss = nullptr, *part = nullptr;
    int* err = nullptr;                       // the device's tensor-core error word
    // tensor maps of k_layer's operands (all of them this object's buffers) for batch mapB
    int mapB = 0;
    CUtensorMap mG, mFT, mT, mDS, mDZ, mH[NLAYER], mWp[NLAYER], mWpT[NLAYER];
};

namespace {

template <typename P>
int alloc0(P** p, size_t bytes) {
    if (cudaMalloc(reinterpret_cast<void**>(p), bytes) != cudaSuccess) return OPTIFAX_ERR_NO_MEMORY;
    if (cudaMemset(*p, 0, bytes) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    return OPTIFAX_OK;
}

#define OFX_TRY(x)                    \
    do {                              \
        int rc_ = (x);                \
        if (rc_) return rc_;          \
    } while (0)

int fno_maps(optifax_fno_s* f, int B) {
    if (f->mapB == B) return OPTIFAX_OK;
    f->mapB = 0;
    const long long L = f->L, BL = (long long)B * L;
    for (int l = 1; l < NLAYER; ++l) {
        f->S[l] = f->S[0] + (long long)l * B * W * SPEC;
        f->dT[l] = f->dT[0] + (long long)l * B * W * SPEC;
    }
    OFX_TRY(ofx_tc::make_map(&f->mG, f->G, L, SPEC, SPEC, 128));
    OFX_TRY(ofx_tc::make_map(&f->mFT, f->FT, L, SPEC, SPEC, 128));
    OFX_TRY(ofx_tc::make_map(&f->mT, f->T, (long long)B * W, SPEC, SPEC, 64));
    OFX_TRY(ofx_tc::make_map(&f->mDS, f->dS, (long long)B * W, SPEC, SPEC, 64));
    OFX_TRY(ofx_tc::make_map(&f->mDZ, f->dZt, BL, W, W, 128));
    for (int l = 0; l < NLAYER; ++l) {
        OFX_TRY(ofx_tc::make_map(&f->mH[l], f->Ht[l], BL, W, W, 128));
        OFX_TRY(ofx_tc::make_map(&f->mWp[l], f->wb + off_wp(l), W, W, W, 64));
        OFX_TRY(ofx_tc::make_map(&f->mWpT[l], f->wpt + (long long)l * W * W, W, W, W, 64));
    }
    f->mapB = B;
    return OPTIFAX_OK;
}

// K splits of the transform products (M = 64 B rows, K = L).  Their FP32 sums are rounded
// to BF16 behind the mixing, so the number is part of the result and the same for every
// batch.
constexpr int SPEC_SPLITS = 8;

int fno_forward(optifax_fno_s* f, const float* x, float* y, int B, cudaStream_t st) {
    const int L = f->L;
    const long long WB = (long long)W * B, rowsA = WB > 128 ? WB : 128;
    OFX_TRY(fno_maps(f, B));
    // the split-K products add into S: one clearing for the four layers
    if (cudaMemsetAsync(f->S[0], 0, sizeof(float) * NLAYER * WB * SPEC, st) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    launch_dep(k_lift, dim3(nblk((long long)B * L, 64)), dim3(256), 0, st, x, f->wb + OFF_P, f->master + OFF_PB, B, L,
               f->Hc[0], f->Ht[0]);
    for (int l = 0; l < NLAYER; ++l) {
        OFX_TRY(optifax_gemm_bf16(f->Hc[l], L, rowsA, f->F, L, SPEC, f->S[l], SPEC, (int)WB, SPEC, L,
                                  SPEC_SPLITS, 1, st));
        launch_mix<false>(f->S[l], f->wb + off_ws(l), B, f->T, st);
        LayerArgs a = {};
        a.bias = f->master + off_b(l);
        a.act = l < NLAYER - 1;
        a.Z = a.act ? f->Z[l] : nullptr;
        a.Hc = f->Hc[l + 1]; a.Ht = f->Ht[l + 1];
        a.err = f->err; a.B = B; a.L = L;
        launch_dep(k_layer<LAYER_FWD>, dim3((L + 127) / 128, B), dim3(128), LAYER_SMEM, st, f->mG, f->mH[l], f->mT,
                   f->mWp[l], a);
    }
    launch_dep(k_proj_fwd, dim3(nblk((long long)B * L, 64)), dim3(256), 0, st, f->Ht[NLAYER], f->wb + OFF_Q,
               f->master + OFF_QB, x, B, L, y);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

int fno_backward(optifax_fno_s* f, const float* x, const float* target, const float* sample_w, int B,
                 cudaStream_t st) {
    const int L = f->L;
    const long long WB = (long long)W * B, BL = (long long)B * L;
    if (cudaMemsetAsync(f->grad, 0, sizeof(float) * N_PARAMS, st) != cudaSuccess ||
        cudaMemsetAsync(f->dT[0], 0, sizeof(float) * NLAYER * WB * SPEC, st) != cudaSuccess ||
        cudaMemsetAsync(f->loss, 0, sizeof(float), st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    const long long ny = BL * COUT;
    launch_dep(k_loss, dim3(256), dim3(256), 0, st, f->y, target, sample_w, (long long)COUT * L, ny, 1.f / (float)ny,
               f->dy, f->loss);
    launch_dep(k_proj_bwd, dim3((L + 255) / 256, B), dim3(256), 0, st, f->dy, f->wb + OFF_Q, f->Ht[NLAYER], B, L, f->dZc,
               f->dZt, f->grad + off_b(NLAYER - 1), f->grad + OFF_Q, f->grad + OFF_QB);
    for (int l = NLAYER - 1; l >= 0; --l) {
        // dWp: K = B L over CTAs of 512 (64 rows of A: half of the tile is padding)
        const int splits = (int)(BL <= (4096LL << 9) ? (BL + 511) / 512 : 4096);
        OFX_TRY(optifax_gemm_bf16(f->dZc, BL, 128, f->Hc[l], BL, W, f->grad + off_wp(l), W, W, W, (int)BL, splits, 1,
                                  st));
        OFX_TRY(optifax_gemm_bf16(f->dZc, L, 2 * WB, f->GT, L, SPEC, f->dT[l], SPEC, (int)WB, SPEC, L,
                                  SPEC_SPLITS, 1, st));
        launch_mix<true>(f->dT[l], f->wb + off_ws(l), B, f->dS, st);
        launch_dep(k_mix_bwd_dw, dim3(nblk((long long)W * W * MODES)), dim3(256), 0, st, f->dT[l], f->S[l], B,
                   f->grad + off_ws(l));
        LayerArgs a = {};
        a.err = f->err; a.B = B; a.L = L;
        const dim3 grid((L + 127) / 128, B);
        if (l > 0) {
            a.Z = f->Z[l - 1];
            a.Hc = f->dZc; a.Ht = f->dZt;
            a.db = f->grad + off_b(l - 1);
            launch_dep(k_layer<LAYER_BWD>, grid, dim3(128), LAYER_SMEM, st, f->mFT, f->mDZ, f->mDS, f->mWpT[l], a);
        } else {
            a.x = x;
            a.db = f->part;
            launch_dep(k_layer<LAYER_BWD_IN>, grid, dim3(128), LAYER_SMEM, st, f->mFT, f->mDZ, f->mDS, f->mWpT[l], a);
            launch_dep(k_lift_sum, dim3(W * 8 / 32, 8), dim3(256), 0, st, f->part, (int)(grid.x * grid.y),
                       f->grad + OFF_P, f->grad + OFF_PB);
        }
    }
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

void fno_free(optifax_fno_s* f) {
    void* ps[] = {f->master, f->grad, f->m, f->v, f->wb, f->wpt, f->F, f->FT, f->G, f->GT, f->T, f->dS, f->dZc,
                  f->dZt, f->y, f->dy, f->loss, f->part};
    for (void* p : ps)
        if (p) cudaFree(p);
    for (int l = 0; l <= NLAYER; ++l) {
        if (f->Hc[l]) cudaFree(f->Hc[l]);
        if (f->Ht[l]) cudaFree(f->Ht[l]);
    }
    if (f->S[0]) cudaFree(f->S[0]);
    if (f->dT[0]) cudaFree(f->dT[0]);
    for (int l = 0; l < NLAYER - 1; ++l)
        if (f->Z[l]) cudaFree(f->Z[l]);
    delete f;
}

}  // namespace

extern "C" int64_t optifax_fno_param_count(void) { return N_PARAMS; }

extern "C" int optifax_fno_create(optifax_fno* out, int32_t n_bins, int32_t max_batch, int32_t device) {
    if (!out) return OPTIFAX_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (n_bins < 128 || n_bins % 64 || n_bins > (1 << 20) || max_batch < 1 || max_batch > 4096)
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    optifax_fno_s* f = new optifax_fno_s();
    f->device = device;
    f->L = n_bins;
    f->maxB = max_batch;
    const long long L = n_bins, WB = (long long)W * max_batch, rowsA = WB > 128 ? WB : 128, BL = max_batch * L;
    int rc = OPTIFAX_OK;
    auto A = [&](auto** p, size_t bytes) {
        if (!rc) rc = alloc0(p, bytes);
    };
    A(&f->master, sizeof(float) * N_PARAMS);
    A(&f->grad, sizeof(float) * N_PARAMS);
    A(&f->m, sizeof(float) * N_PARAMS);
    A(&f->v, sizeof(float) * N_PARAMS);
    A(&f->wb, sizeof(bf16) * N_PARAMS);
    A(&f->wpt, sizeof(bf16) * NLAYER * W * W);
    A(&f->F, sizeof(bf16) * SPEC * L);
    A(&f->FT, sizeof(bf16) * SPEC * L);
    A(&f->G, sizeof(bf16) * SPEC * L);
    A(&f->GT, sizeof(bf16) * SPEC * L);
    for (int l = 0; l <= NLAYER; ++l) {
        A(&f->Hc[l], sizeof(bf16) * rowsA * L);
        A(&f->Ht[l], sizeof(bf16) * BL * W);
    }
    for (int l = 0; l < NLAYER - 1; ++l) A(&f->Z[l], sizeof(float) * WB * L);
    A(&f->S[0], sizeof(float) * NLAYER * WB * SPEC);
    A(&f->dT[0], sizeof(float) * NLAYER * WB * SPEC);
    A(&f->part, sizeof(float) * W * 8 * max_batch * ((L + 127) / 128));
    A(&f->T, sizeof(bf16) * rowsA * SPEC);
    A(&f->dS, sizeof(bf16) * rowsA * SPEC);
    A(&f->dZc, sizeof(bf16) * 2 * WB * L);     // the [o][(b,x)] view is read as 128 rows
    A(&f->dZt, sizeof(bf16) * BL * W);
    A(&f->y, sizeof(float) * BL * COUT);
    A(&f->dy, sizeof(float) * BL * COUT);
    A(&f->loss, sizeof(float));
    if (!rc) {
        f->err = ofx_tc::error_word();
        if (!f->err ||
            cudaFuncSetAttribute(k_layer<LAYER_FWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, LAYER_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_layer<LAYER_BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, LAYER_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_layer<LAYER_BWD_IN>, cudaFuncAttributeMaxDynamicSharedMemorySize, LAYER_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_mix<false, MIXU, MIXB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Mix<MIXU, MIXB>::smem) != cudaSuccess ||
            cudaFuncSetAttribute(k_mix<true, MIXU, MIXB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Mix<MIXU, MIXB>::smem) != cudaSuccess)
            rc = OPTIFAX_ERR_CUDA;
    }
    if (!rc) {
        k_dft_tables<<<nblk((long long)SPEC * L), 256>>>((int)L, f->F, f->FT, f->G, f->GT);
        if (cudaDeviceSynchronize() != cudaSuccess) rc = OPTIFAX_ERR_CUDA;
    }
    if (rc) {
        fno_free(f);
        return rc;
    }
    *out = f;
    return OPTIFAX_OK;
}

extern "C" int optifax_fno_destroy(optifax_fno f) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    cudaSetDevice(f->device);
    cudaDeviceSynchronize();
    fno_free(f);
    return OPTIFAX_OK;
}

extern "C" int optifax_fno_set_params(optifax_fno f, const float* params, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (!params) return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(f->master, params, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(f->m, 0, sizeof(float) * N_PARAMS, st) != cudaSuccess ||
        cudaMemsetAsync(f->v, 0, sizeof(float) * N_PARAMS, st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    k_refresh<<<nblk(N_PARAMS), 256, 0, st>>>(f->master, f->wb, f->wpt);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_fno_get_params(optifax_fno f, float* params, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (!params) return OPTIFAX_ERR_INVALID_ARGUMENT;
    return cudaMemcpyAsync(params, f->master, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToDevice,
                           static_cast<cudaStream_t>(stream)) == cudaSuccess
               ? OPTIFAX_OK
               : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_fno_forward(optifax_fno f, const float* x, float* y, int32_t batch, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (!x || batch < 1 || batch > f->maxB) return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the network reads x to its end: an output that lies over the input is written last
    const size_t nx = (size_t)batch * CIN * f->L, ny = (size_t)batch * COUT * f->L;
    const bool apart = y && (y + ny <= x || x + nx <= y);
    OFX_TRY(fno_forward(f, x, apart ? y : f->y, batch, st));
    if (y && !apart &&
        cudaMemcpyAsync(y, f->y, sizeof(float) * ny, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    return OPTIFAX_OK;
}

extern "C" int optifax_fno_backward(optifax_fno f, const float* x, const float* target, const float* sample_w,
                                    int32_t batch, float* loss, float* grads, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (!x || !target || batch < 1 || batch > f->maxB) return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    OFX_TRY(fno_forward(f, x, f->y, batch, st));
    OFX_TRY(fno_backward(f, x, target, sample_w, batch, st));
    if (loss && cudaMemcpyAsync(loss, f->loss, sizeof(float), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    if (grads && cudaMemcpyAsync(grads, f->grad, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    return OPTIFAX_OK;
}

// Data-parallel training: replace the gradients of the last backward (for example by
// their mean over ranks) before optifax_fno_adam.
extern "C" int optifax_fno_set_grads(optifax_fno f, const float* grads, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (!grads) return OPTIFAX_ERR_INVALID_ARGUMENT;
    return cudaMemcpyAsync(f->grad, grads, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToDevice,
                           static_cast<cudaStream_t>(stream)) == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_fno_adam(optifax_fno f, float lr, float beta1, float beta2, float eps, float weight_decay,
                                int32_t step, void* stream) {
    if (!f) return OPTIFAX_ERR_NULL_HANDLE;
    if (step < 1 || !(lr >= 0.f)) return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float bc1 = 1.f - powf(beta1, (float)step), bc2 = 1.f - powf(beta2, (float)step);
    k_adam<<<nblk(N_PARAMS), 256, 0, st>>>(f->master, f->grad, f->m, f->v, N_PARAMS, lr, beta1, beta2, eps,
                                           weight_decay, bc1, bc2);
    k_refresh<<<nblk(N_PARAMS), 256, 0, st>>>(f->master, f->wb, f->wpt);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_ff_encode(const void* spectra, int64_t stride, int32_t n_spectra, int32_t n_points, int32_t k0,
                                 int32_t n_bins, int32_t split, float pump_scale, const float* sigma_in, float* x,
                                 int32_t n_channels, float* sigma_out, void* stream) {
    if (!spectra || !x || n_spectra < 1 || n_points < 1 || n_bins < 1 || n_bins > n_points || k0 < 0 ||
        k0 >= n_points || split < 0 || split > n_bins || stride < n_points || !(pump_scale > 0.f) ||
        (n_channels != 4 && n_channels != 6))
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    k_ff_encode<<<n_spectra, 1024, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(spectra), stride, n_points, k0, n_bins, split, pump_scale, sigma_in, x, n_channels,
        sigma_out);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_ff_step(const float* y, const float* sigma, const void* X_in, const void* feedback,
                               const void* pump, const void* lin, const float* tally_w, int32_t n_points, int32_t k0,
                               int32_t n_bins, int32_t split, float pump_scale, void* X_out, void* Y_next,
                               double* energy, void* stream) {
    if ((!y && !X_in) || (y && !sigma) || !feedback || !pump || !Y_next || n_points < 1 || n_bins < 1 ||
        n_bins > n_points || k0 < 0 || k0 >= n_points || split < 0 || split > n_bins || !(pump_scale > 0.f))
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (energy && cudaMemsetAsync(energy, 0, sizeof(double), st) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    launch_dep(k_ff_step, dim3(nblk(n_points)), dim3(256), 0, st, y, sigma, static_cast<const float2*>(X_in),
               static_cast<const float2*>(feedback), static_cast<const float2*>(pump), static_cast<const float2*>(lin),
               tally_w, (int)n_points, (int)k0, (int)n_bins, (int)split, pump_scale, static_cast<float2*>(X_out),
               static_cast<float2*>(Y_next), energy);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

namespace {
int env_args(int32_t n_points, int32_t n_bins, const int32_t* band, EnvBand* bp, EnvBand* bs, int* logL) {
    if (!band || n_points < 1 || n_bins < 2 || n_bins > 4096 || (n_bins & (n_bins - 1)) || n_bins > n_points)
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    *bp = {band[0], band[1], band[2]};
    *bs = {band[3], band[4], band[5]};
    for (const EnvBand* b : {bp, bs})
        if (b->kc < 0 || b->kc >= n_points || b->lo < -n_bins / 2 || b->hi > n_bins / 2 || b->lo >= b->hi)
            return OPTIFAX_ERR_INVALID_ARGUMENT;
    int l = 0;
    while ((1 << l) < n_bins) ++l;
    *logL = l;
    return OPTIFAX_OK;
}
}  // namespace

extern "C" int optifax_ff_encode_env(const void* spectra, int64_t stride, int32_t n_spectra, int32_t n_points,
                                     int32_t n_bins, const int32_t* band, float pump_scale, const float* sigma_in,
                                     float* x, int32_t n_channels, float* sigma_out, void* stream) {
    EnvBand bp, bs;
    int logL = 0;
    if (!spectra || !x || n_spectra < 1 || stride < n_points || !(pump_scale > 0.f) ||
        (n_channels != 4 && n_channels != 6))
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    int rc = env_args(n_points, n_bins, band, &bp, &bs, &logL);
    if (rc) return rc;
    launch_dep(k_ff_encode_env, dim3(n_spectra, 2), dim3(ENV_T), 0, static_cast<cudaStream_t>(stream),
               static_cast<const float2*>(spectra), (long long)stride, (int)n_points, (int)n_bins, logL, bp, bs,
               pump_scale, sigma_in, x, (int)n_channels, sigma_out);
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

extern "C" int optifax_ff_decode_env(const float* y, const float* sigma, int32_t n_points, int32_t n_bins,
                                     const int32_t* band, float pump_scale, void* X_out, void* stream) {
    EnvBand bp, bs;
    int logL = 0;
    if (!y || !sigma || !X_out || !(pump_scale > 0.f)) return OPTIFAX_ERR_INVALID_ARGUMENT;
    int rc = env_args(n_points, n_bins, band, &bp, &bs, &logL);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    launch_dep(k_ff_decode_env, dim3(2 + nblk(n_points, ENV_T)), dim3(ENV_T), 0, st, y, sigma, (int)n_points,
               (int)n_bins, logL, bp, bs, pump_scale, static_cast<float2*>(X_out));
    return cudaGetLastError() == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}
