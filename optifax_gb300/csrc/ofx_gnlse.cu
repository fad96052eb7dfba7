// ofx_gnlse.cu -- chi(3) fibre GNLSE on the GPU: one persistent CTA per pulse.
//
// Replaces toolbox/lib/internal/main/gnlsefib.m:1-89.  The interaction-picture
// spectral field AW (n modes, FFT order) obeys gnlsefib.m:54-66,
//     dAW/dz = i gamma W ifft(AT ((1 - fR)|AT|^2 + RS)) e^{-Lz},
//     AT = fft(AW e^{Lz}),  RS = dT fR fft(ifft(|AT|^2) RW),  L = iB - alpha/2,
// in MATLAB's fft/ifft conventions (fft: exp(-i), ifft: exp(+i)/n), from
// AW(0) = ifft(A).  The reference integrates it with MATLAB's ode45 (RelTol,
// AbsTol, NormControl; gnlsefib.m:77-80), outputs at linspace(0, L, n_saves).
// Here: the Dormand-Prince 5(4) pair with the same tolerances and error norm,
//     err = ||h sum_i e_i k_i|| / max(||y||, ||y_new||, AbsTol/RelTol) <= RelTol,
// under ode45's published step control (Shampine & Reichelt 1997): initial step
// min(L/10, 0.8 RelTol^(1/5) max(||y0||, thr) / ||f0||), steps of at most L/10
// stretched to the end when 1.1 h reaches it, a first failure scaling h by
// max(0.1, 0.8 (RelTol/err)^(1/5)) and later ones halving it, growth by
// min(5, 0.8 (RelTol/err)^(1/5)) only after a step that did not fail.  Steps do
// not stop at the save points: a save point inside an accepted step is output
// from a separate step of exactly that length from the step's start (its stages
// reuse the accepted step's k1 and rows k2..k6; y_new waits in an eighth scratch
// row).  Positions are integers in units of length / 2^40 so that every
// dispersion phase B_k z is a 64-bit fixed-point product (exact mod one turn; only
// the final angle goes
// through FP32).  FP32 field arithmetic, norms reduced across the CTA in FP64
// (per-thread partials of 4 or 8 modes in FP32), FP64 step control.
//
// Layout: the CTA's M/P threads hold the spectral state y in registers, P modes each
// (8, or 4 below 2048 points), in the FFT's bit-reversed slot order (slot s <-> mode
// bitrev(s)); the seven stage derivatives k_i and y_new sit in an L2-resident global
// scratch (8 x n per pulse, each thread touching only its own values, laid out so that a
// warp's loads are contiguous).  Each right-hand side costs four in-place M-point
// transforms (two without Raman): MATLAB's fft of a spectral array is
// conj(inverse(conj(.))), its ifft (1/n) conj(forward(conj(.))).  The point-wise steps in
// the time domain work on the registers between the last pass of an inverse and the
// first pass of the next forward transform, so one shared-memory buffer serves all four.
// Stages 2, 4 and 6 read the rows once for two sums, their own and the next stage's (the
// error's), which waits in shared memory for its last term: 9 rows read a step, not 26.
// What bounds it: the serial chain of 24 transforms a step on one SM per pulse (2,500 to
// 3,500 cycles each at 4096 points).
#include <cmath>
#include <cstdint>

#include "ofx_fft.cuh"
#include "ofx_gnlse.cuh"

namespace ofx {
namespace {

constexpr int kZBits = 40;

// Dormand-Prince 5(4) tableau (Dormand & Prince 1980): nodes here; stage weights
// (row 6 = the 5th-order weights, FSAL) and error weights b - b_hat below (kA, kE).
__constant__ double kDpC[7] = {0.0, 1.0 / 5, 3.0 / 10, 4.0 / 5, 8.0 / 9, 1.0, 1.0};

__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// Squared norm of a thread's modes: FP32 partial sums (8 terms, relative error below 1e-6)
template <int P>
__device__ __forceinline__ float norm2(const float2 (&a)[P]) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < P; ++j) s = fmaf(a[j].x, a[j].x, fmaf(a[j].y, a[j].y, s));
    return s;
}

// Sums of two per-thread values over the CTA in FP64 (part: 2 T floats, red: 8 doubles),
// for warp 0 alone.  An FP64 instruction of one warp takes 64 cycles of its scheduler's
// narrow FP64 unit, so the sums are four warps' work, one per scheduler, and every warp
// reducing its own and adding up all warps' (as this was) took 10,000 cycles.
template <int T>
__device__ __forceinline__ void block_sum2(float a, float b, float* part, double* red, double (&out)[2]) {
    const int t = threadIdx.x;
    part[t] = a;
    part[T + t] = b;
    __syncthreads();
    if (t < 128) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < T / 128; ++i) {
            x += (double)part[t + 128 * i];
            y += (double)part[T + t + 128 * i];
        }
        // lanes 0-15 go on with a, 16-31 with b
        const bool up = t & 16;
        double z = (up ? y : x) + __shfl_xor_sync(0xffffffffu, up ? x : y, 16);
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
        if ((t & 15) == 0) red[2 * (t >> 5) + (up ? 1 : 0)] = z;
    }
    __syncthreads();
    if (t < 32) {
        out[0] = (red[0] + red[2]) + (red[4] + red[6]);
        out[1] = (red[1] + red[3]) + (red[5] + red[7]);
    }
}

// Own modes of stage array j in the global scratch: pairs of modes, [pair][thread]
template <int M, int P>
__device__ __forceinline__ void load_row(const float2* K, int j, int t, float2 (&v)[P]) {
    const float4* r = reinterpret_cast<const float4*>(K + (size_t)j * M) + t;
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
        const float4 w = r[i * (M / P)];
        v[2 * i] = make_float2(w.x, w.y);
        v[2 * i + 1] = make_float2(w.z, w.w);
    }
}
template <int M, int P>
__device__ __forceinline__ void store_row(float2* K, int j, int t, const float2 (&v)[P]) {
    float4* r = reinterpret_cast<float4*>(K + (size_t)j * M) + t;
#pragma unroll
    for (int i = 0; i < P / 2; ++i) r[i * (M / P)] = make_float4(v[2 * i].x, v[2 * i].y, v[2 * i + 1].x, v[2 * i + 1].y);
}

// The same tableau as compile-time values, so that the stage combinations unroll
// (all their L2 loads in flight together) and skip the zero weights.
__host__ __device__ constexpr float dp_a(int r, int q) {
    switch (r * 8 + q) {
        case 8: return 1.0f / 5;
        case 16: return 3.0f / 40;
        case 17: return 9.0f / 40;
        case 24: return 44.0f / 45;
        case 25: return -56.0f / 15;
        case 26: return 32.0f / 9;
        case 32: return 19372.0f / 6561;
        case 33: return -25360.0f / 2187;
        case 34: return 64448.0f / 6561;
        case 35: return -212.0f / 729;
        case 40: return 9017.0f / 3168;
        case 41: return -355.0f / 33;
        case 42: return 46732.0f / 5247;
        case 43: return 49.0f / 176;
        case 44: return -5103.0f / 18656;
        case 48: return 35.0f / 384;
        case 50: return 500.0f / 1113;
        case 51: return 125.0f / 192;
        case 52: return -2187.0f / 6784;
        case 53: return 11.0f / 84;
        default: return 0.f;
    }
}
__host__ __device__ constexpr float dp_e(int q) {
    switch (q) {
        case 0: return 71.0f / 57600;
        case 2: return -71.0f / 16695;
        case 3: return 71.0f / 1920;
        case 4: return -17253.0f / 339200;
        case 5: return 22.0f / 525;
        case 6: return -1.0f / 40;
        default: return 0.f;
    }
}

// a += sum_{q < R - 1} a_Rq h k_q and, with the row after it (R2; the error weights when
// R2 < 0), b += sum_{q < R - 1} w_q h k_q from one reading of the rows; then both add
// the k_{R-1} of the registers.  The next stage continues from b.
template <int R, int R2, int M, int P>
__device__ __forceinline__ void combine2(float2 (&a)[P], float2 (&b)[P], const float2 (&last)[P], const float2* K,
                                         int t, int base, float hz) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const float wa = dp_a(R, q), wb = R2 >= 0 ? dp_a(R2, q) : dp_e(q);
        if (wa == 0.f && wb == 0.f) continue;
        float2 k[P];
        if (q < R - 1) load_row<M, P>(K, (base + q) % 7, t, k);
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const float2 kj = q < R - 1 ? k[j] : last[j];
            if (wa != 0.f) a[j] = cfma1(kj, hz * wa, a[j]);
            if (wb != 0.f) b[j] = cfma1(kj, hz * wb, b[j]);
        }
    }
}

// What warp 0 decides and the CTA reads.
struct GCtl {
    double ny, acc_nyn, acc_err;
    long long zc, hc, side_z, save_z;
    long long next_z;                    // position of save point save_idx (past the end: none left)
    long long zs[8];                     // the attempt's stage positions, with e^{-alpha z / 2} and its inverse
    float att[8], iatt[8];
    float hz, save_att;
    int save_idx, save_i, attempts, accepted, status, nofailed, side, base, flags;
};
enum : int { kStash = 1, kAdvance = 2, kSave = 4, kEnd = 8 };

}  // namespace

template <int M>
struct SmemG {
    static constexpr int P = kPoints<M>, T = M / P;
    using F = FftPlan<M, P>;
    static constexpr size_t off_rate = sizeof(float2) * M;                        // B_k z per z unit, 2^-64 turns
    static constexpr size_t off_rw = off_rate + sizeof(uint64_t) * M;
    static constexpr size_t off_w = off_rw + sizeof(float2) * M;
    static constexpr size_t off_tw = off_w + sizeof(float) * M;
    static constexpr size_t off_td = (off_tw + sizeof(float2) * F::TW + 15) & ~size_t(15);
    static constexpr size_t off_part = off_td + sizeof(float) * F::TD;             // sum carried to the next stage
    static constexpr size_t bytes = off_part + sizeof(float2) * M;
};

template <int M>
__global__ void __launch_bounds__(M / kPoints<M>, 1)
gnlse_kernel(const GnlseDev* __restrict__ pulses, const Twiddle* __restrict__ quad) {
    using SM = SmemG<M>;
    constexpr int P = SM::P, T = SM::T;
    constexpr int LOG2M = ilog2(M);
    extern __shared__ __align__(16) unsigned char smem[];
    float2* buf = reinterpret_cast<float2*>(smem);
    uint64_t* rate_s = reinterpret_cast<uint64_t*>(smem + SM::off_rate);
    float2* rw_s = reinterpret_cast<float2*>(smem + SM::off_rw);
    float* w_s = reinterpret_cast<float*>(smem + SM::off_w);
    float2* tw = reinterpret_cast<float2*>(smem + SM::off_tw);
    float* td = reinterpret_cast<float*>(smem + SM::off_td);
    float4* carry = reinterpret_cast<float4*>(smem + SM::off_part);
    float* part = reinterpret_cast<float*>(smem);                         // norms: buf between two transforms
    __shared__ double red[8];
    __shared__ GCtl ctl;

    const int t = threadIdx.x;
    __shared__ GnlseDev sP;
    if (t == 0) sP = pulses[blockIdx.x];
    fft_tables<M, P>(tw, td, quad, t);
    __syncthreads();
    const GnlseDev& P_ = sP;
    const bool raman = (P_.RW != nullptr);
    const double unit = P_.length / (double)(1ll << kZBits);
    const long long total = 1ll << kZBits;
    const long long hmax = total / 10;
    const double thr = P_.atol / P_.rtol, half_loss = 0.5 * P_.alpha;
    const float rtolf = (float)P_.rtol;
    constexpr float invM = 1.0f / (float)M;
    const float gam = (float)P_.gamma, omfr = (float)(1.0 - P_.fr), dtfr = (float)(P_.dT * P_.fr);
    const float awscale = (float)(P_.dT * (double)M);
    float2* K = P_.K;

    // per-mode tables of the own slots (slot s holds mode bitrev(s)), [j][thread]
#pragma unroll 1
    for (int j = 0; j < P; ++j) {
        const int k = bitrev(P * t + j, LOG2M), i = j * T + t;
        double r = P_.B[k] * unit * 0.15915494309189533577;     // turns per z unit
        r -= rint(r);
        double x = r * 18446744073709551616.0;
        if (x >= 9.2233720368547758e18) x -= 1.8446744073709552e19;
        rate_s[i] = (uint64_t)(long long)llrint(x);
        w_s[i] = P_.W[k];
        rw_s[i] = raman ? P_.RW[k] : make_float2(0.f, 0.f);
    }
    // y(0) = ifft(A) = conj(forward(conj(A))) / M
    float2 y[P], ys[P], v[P], e[P];
#pragma unroll
    for (int q = 0; q < P; ++q) v[q] = conjf2(P_.A[t + q * T]);
    fftp_forward_regs<M, P>(buf, tw, t, v);
#pragma unroll
    for (int j = 0; j < P; ++j) y[j] = cscale(conjf2(v[j]), invM);

    const long long nm1 = P_.n_saves - 1;
    auto save_point = [&](int i) -> long long {
        return i < P_.n_saves ? ((long long)i * total + nm1 / 2) / nm1 : total + 1;
    };

    // ---- control: warp 0, all lanes the same values, lane 0 writes ----
    // The scalar FP64 arithmetic of a step in every warp cost a third of the step (a warp's
    // FP64 instruction occupies the scheduler's unit for 64 cycles).
    // Positions and attenuations of the next attempt's stages, one per lane; side: a step to side_z
    auto prepare = [&](bool side) {
        const int stage = t < 7 ? t : 6;
        const long long span = side ? ctl.side_z - ctl.zc : ctl.hc;
        const long long zs = stage == 0 ? (side ? ctl.side_z : ctl.zc) : ctl.zc + llrint(kDpC[stage] * (double)span);
        const double zd = (double)zs * unit;
        const float loss = (float)(half_loss * zd), att = expf(-loss), iatt = expf(loss);
        const float hz = (float)((double)span * unit);
        __syncwarp();
        if (t < 7) {
            ctl.zs[t] = zs;
            ctl.att[t] = att;
            ctl.iatt[t] = iatt;
        }
        if (t == 0) {
            ctl.hz = hz;
            ctl.side = side;
            if (side) {
                const int i = ctl.save_idx;
                ctl.save_i = i;
                ctl.save_idx = i + 1;
                ctl.next_z = save_point(i + 1);
                ctl.save_z = zs;
                ctl.save_att = att;
            }
        }
        __syncwarp();
    };
    auto new_step = [&](long long h) {                 // a first attempt with step h
        h = h > hmax ? hmax : (h < 1 ? 1 : h);
        long long hc = h;
        const long long left = total - ctl.zc;
        if (1.1 * (double)hc >= (double)left) hc = left;                   // stretch to the end
        __syncwarp();
        if (t == 0) { ctl.hc = hc; ctl.nofailed = 1; }
        __syncwarp();
        prepare(false);
    };
    auto side_step = [&]() -> bool {                   // the next save point, if inside the accepted step
        const long long z = ctl.next_z;
        const bool in = z < ctl.zc + ctl.hc;
        __syncwarp();
        if (in) {
            if (t == 0) ctl.side_z = z;
            __syncwarp();
            prepare(true);
        }
        return in;
    };
    auto advance = [&]() -> int {                      // the accepted step becomes the state
        const long long hc = ctl.hc, zc = ctl.zc + hc;
        const double err = ctl.acc_err;
        const bool save = ctl.next_z == zc;
        const int i = ctl.save_idx + (save ? 1 : 0), flags = save ? kAdvance | kSave : kAdvance;
        const bool nofailed = ctl.nofailed, limit = ctl.attempts >= P_.max_attempts;
        __syncwarp();
        if (t == 0) {
            ctl.zc = zc;
            ctl.ny = ctl.acc_nyn;
            ctl.base = (ctl.base + 6) % 7;             // FSAL: k7 becomes the next k1
            if (save) {
                ctl.save_i = i - 1;
                ctl.save_z = zc;
                ctl.save_att = expf(-(float)(half_loss * ((double)zc * unit)));
                ctl.save_idx = i;
                ctl.next_z = save_point(i);
            }
        }
        __syncwarp();
        if (i >= P_.n_saves || zc >= total) return flags | kEnd;
        // growth after a step with no failure: h / (1.25 (err/rtol)^(1/5)), at most 5 h
        long long h = hc;
        if (nofailed) {
            const float temp = 1.25f * powf((float)(err / P_.rtol), 0.2f);
            h = temp > 0.2f ? (long long)((double)hc / (double)temp) : 5 * hc;
        }
        if (limit) {
            if (t == 0) ctl.status |= OPTIFAX_PULSE_ATTEMPT_LIMIT;
            return flags | kEnd;
        }
        new_step(h);
        return flags;
    };
    auto decide = [&](const double (&s2)[2]) -> int {  // after the last stage of an attempt
        const double root = sqrt((t & 1) ? s2[1] : s2[0]);
        const double errn = __shfl_sync(0xffffffffu, root, 0), nyn = __shfl_sync(0xffffffffu, root, 1);
        const double err = errn / fmax(fmax(ctl.ny, nyn), thr);
        const bool ok = err <= P_.rtol;
        const int attempts = ctl.attempts;
        const long long hc = ctl.hc;
        const bool nofailed = ctl.nofailed, nan = !isfinite(errn) || !isfinite(nyn);
        __syncwarp();
        if (t == 0) {
            if (P_.trace && attempts < P_.trace_cap) {
                P_.trace[2 * attempts] = hc;
                P_.trace[2 * attempts + 1] = ok ? 1 : 0;
            }
            ctl.attempts = attempts + 1;
            if (nan) ctl.status |= OPTIFAX_PULSE_NAN;
            else if (ok) {
                ++ctl.accepted;
                ctl.acc_err = err;
                ctl.acc_nyn = nyn;
            }
        }
        __syncwarp();
        if (nan) return kEnd;
        // a save point inside the step: y_new is stashed, then a step of exactly that length
        if (ok) return side_step() ? kStash : advance();
        // a failed step: the first failure scales by max(0.1, 0.8 (rtol/err)^(1/5)),
        // later ones halve (the factor only scales an integer step: FP32 powf serves)
        long long next = hc / 2;
        if (nofailed) {
            next = (long long)((double)hc * (double)fmaxf(0.1f, 0.8f * powf(rtolf / (float)err, 0.2f)));
        }
        if (t == 0) {
            ctl.nofailed = 0;
            ctl.hc = next < 1 ? 1 : next;
        }
        __syncwarp();
        if (attempts + 1 >= P_.max_attempts) {
            if (t == 0) ctl.status |= OPTIFAX_PULSE_ATTEMPT_LIMIT;
            return kEnd;
        }
        prepare(false);
        return 0;
    };

    // save ctl.save_i from the spectral state src at position ctl.save_z: AW e^{Lz}
    // (fftshifted, x dT n) and AT = fft(AW e^{Lz})
    auto do_save = [&](const float2 (&src)[P]) {
        const float att = ctl.save_att;
        const uint64_t zp = (uint64_t)ctl.save_z;
        const size_t row = (size_t)ctl.save_i * M;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const float2 aw = cscale(cmul(src[j], turn_to_unit(rate_s[j * T + t] * zp)), att);
            const int k = bitrev(P * t + j, LOG2M);
            P_.AW_out[row + ((k + M / 2) & (M - 1))] = cscale(aw, awscale);
            v[j] = conjf2(aw);
        }
        fftp_inverse<M, P>(buf, tw, td, t, v);
#pragma unroll
        for (int q = 0; q < P; ++q) P_.AT_out[row + t + q * T] = conjf2(v[q]);
        __syncthreads();                   // the next transform writes what others may still read
    };
    if (t == 0) {
        ctl = GCtl{};
        ctl.att[0] = ctl.iatt[0] = ctl.save_att = 1.f;
        ctl.save_idx = 1;
        ctl.next_z = save_point(1);
    }
    __syncthreads();
    do_save(y);

    int stage = 0, base = 0, side = 0;
    for (;;) {
        // ---- stage input ys: every second stage reads the rows for itself and the next.  The
        // weighted rows are summed by themselves and y is added last: one rounding at y's size
        // (fields at 4096 points and 1 to 10 kW against FP64 on the same steps: 3.0e-7 with the rows
        // added to y one after the other, 2.6e-7 so) ----
        const float hz = ctl.hz;
        float2 part2[P];                   // the next stage's sum without its last term (stage 6: the error's)
        if (stage == 1) {
            float2 k[P];
            load_row<M, P>(K, base, t, k);
#pragma unroll
            for (int j = 0; j < P; ++j) ys[j] = cfma1(k[j], hz * dp_a(1, 0), y[j]);
        } else if (stage == 3 || stage == 5) {
            const float w = hz * (stage == 3 ? dp_a(3, 2) : dp_a(5, 4));
#pragma unroll
            for (int i = 0; i < P / 2; ++i) {
                const float4 c = carry[i * T + t];
                ys[2 * i] = add2(y[2 * i], cfma1(v[2 * i], w, make_float2(c.x, c.y)));
                ys[2 * i + 1] = add2(y[2 * i + 1], cfma1(v[2 * i + 1], w, make_float2(c.z, c.w)));
            }
        } else if (stage == 0) {
#pragma unroll
            for (int j = 0; j < P; ++j) ys[j] = y[j];
        } else {
#pragma unroll
            for (int j = 0; j < P; ++j) ys[j] = part2[j] = make_float2(0.f, 0.f);
            if (stage == 2) combine2<2, 3, M, P>(ys, part2, v, K, t, base, hz);
            else if (stage == 4) combine2<4, 5, M, P>(ys, part2, v, K, t, base, hz);
            else combine2<6, -1, M, P>(ys, part2, v, K, t, base, hz);
#pragma unroll
            for (int j = 0; j < P; ++j) ys[j] = add2(y[j], ys[j]);
#pragma unroll
            for (int i = 0; i < P / 2; ++i)
                carry[i * T + t] = make_float4(part2[2 * i].x, part2[2 * i].y, part2[2 * i + 1].x, part2[2 * i + 1].y);
        }
        int flags = 0;
        if (stage == 6 && side) {
            // stages k2..k6 of the step to the save point done: y(side_z) = y + h' sum a_7j k_j
            do_save(ys);
            if (t < 32) {
                const int f = side_step() ? 0 : advance();
                if (t == 0) {
                    if (f) ctl.side = 0;
                    ctl.flags = f;
                }
            }
            __syncthreads();
            flags = ctl.flags;
            if (flags & kAdvance) load_row<M, P>(K, 7, t, ys);       // back to the accepted step
        } else {
            // ---- right-hand side f(zs, ys) (gnlsefib.m:54-66) into v ----
            {
                const uint64_t zs = (uint64_t)ctl.zs[stage];
                const float att = ctl.att[stage], iatt = ctl.iatt[stage];
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    if (stage != 6) e[j] = turn_to_unit(rate_s[j * T + t] * zs);   // e^{i B z}; stage 5's position
                    v[j] = conjf2(cscale(cmul(ys[j], e[j]), att));
                }
                fftp_inverse<M, P>(buf, tw, td, t, v);                        // conj(AT)
                float2 at[P];
#pragma unroll
                for (int q = 0; q < P; ++q) at[q] = conjf2(v[q]);
                if (raman) {
#pragma unroll
                    for (int q = 0; q < P; ++q) v[q] = make_float2(at[q].x * at[q].x + at[q].y * at[q].y, 0.f);
                    fftp_forward_regs<M, P>(buf, tw, t, v);                   // forward(|AT|^2)
#pragma unroll
                    for (int j = 0; j < P; ++j)                               // conj(ifft(|AT|^2) RW)
                        v[j] = conjf2(cscale(cmul(conjf2(v[j]), rw_s[j * T + t]), invM));
                    fftp_inverse<M, P>(buf, tw, td, t, v);                    // conj(RS / (dT fR))
                }
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    const float it = at[q].x * at[q].x + at[q].y * at[q].y;
                    const float2 g = raman ? make_float2(fmaf(omfr, it, dtfr * v[q].x), -dtfr * v[q].y)
                                           : make_float2(it, 0.f);
                    v[q] = conjf2(cmul(at[q], g));                            // conj(Q)
                }
                fftp_forward_regs<M, P>(buf, tw, t, v);                       // ifft(Q) = conj(v) / M
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const float2 m = cmul(conjf2(v[j]), conjf2(e[j]));
                    const float s = gam * w_s[j * T + t] * iatt * invM;
                    v[j] = make_float2(-m.y * s, m.x * s);                    // i gamma W M e^{-Lz}
                }
            }
            if (stage != 5) store_row<M, P>(K, (base + stage) % 7, t, v);     // k6 stays in registers
            if (stage > 0 && stage < 6) { ++stage; continue; }
            double s2[2];
            __syncthreads();                   // buf is free for the norms
            if (stage == 0) {
                // initial step (ode45, NormControl): min(hmax, 0.8 rtol^(1/5) max(||y||, thr) / ||f||)
                block_sum2<T>(norm2(y), norm2(v), part, red, s2);
                if (t < 32) {
                    const double ny = sqrt(s2[0]), nf = sqrt(s2[1]);
                    long long h = hmax;
                    if (nf != 0.0) {
                        const double hh = (0.8 * pow(P_.rtol, 0.2)) * fmax(ny, thr) / nf / unit;
                        const long long hi = hh >= (double)hmax ? hmax : (long long)hh;
                        h = hi < 1 ? 1 : hi;
                    }
                    if (t == 0) ctl.ny = ny;
                    new_step(h);
                }
                __syncthreads();
                stage = 1;
                continue;
            }
            // ---- stage 6 done: ys = y_new, error estimate and decision ----
            float2 ev[P];
#pragma unroll
            for (int i = 0; i < P / 2; ++i) {
                const float4 c = carry[i * T + t];
                ev[2 * i] = cfma1(v[2 * i], hz * dp_e(6), make_float2(c.x, c.y));
                ev[2 * i + 1] = cfma1(v[2 * i + 1], hz * dp_e(6), make_float2(c.z, c.w));
            }
            block_sum2<T>(norm2(ev), norm2(ys), part, red, s2);
            if (t < 32) {
                const int f = decide(s2);
                if (t == 0) ctl.flags = f;
            }
            __syncthreads();
            flags = ctl.flags;
            if (flags & kStash) store_row<M, P>(K, 7, t, ys);
        }
        if (flags & kAdvance) {
            base = ctl.base;
#pragma unroll
            for (int j = 0; j < P; ++j) y[j] = ys[j];
            if (flags & kSave) do_save(y);
        }
        if (flags & kEnd) break;
        side = ctl.side;
        stage = 1;
    }
    if (t == 0 && P_.stats) {
        optifax_gnlse_stats st;
        st.attempts = ctl.attempts; st.accepted = ctl.accepted; st.status = ctl.status; st.reserved = 0;
        *P_.stats = st;
    }
}

template <int M>
cudaError_t launch_one(const GnlseDev* d, int n_pulses, const Twiddle* quad, cudaStream_t st) {
    constexpr size_t smem = SmemG<M>::bytes;
    cudaError_t e = cudaFuncSetAttribute(gnlse_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    gnlse_kernel<M><<<n_pulses, SmemG<M>::T, smem, st>>>(d, quad);
    return cudaGetLastError();
}

cudaError_t launch_gnlse(int M, const GnlseDev* d, int n_pulses, const Twiddle* quad, cudaStream_t st) {
    switch (M) {
        case 512: return launch_one<512>(d, n_pulses, quad, st);
        case 1024: return launch_one<1024>(d, n_pulses, quad, st);
        case 2048: return launch_one<2048>(d, n_pulses, quad, st);
        case 4096: return launch_one<4096>(d, n_pulses, quad, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ofx
