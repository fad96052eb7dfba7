// ofx_passx_host.cuh -- host driver of the wide-state crystal pass (ofx_passx.cuh),
// shared by optifax_propagate_fp64 (R = double, ofx_fp64.cu) and
// optifax_propagate_f32x2 (R = float-float, ofx_f32x2.cu).
//
// Interface of both entries: the reference's MEX argument list with double
// arrays (E N x B complex, alpha and beta N, G S or S x B), every pulse of the
// call on one adaptive step schedule (the reference's batch rule, error flags
// OR-ed over the batch through a grid barrier of a cooperative launch), the
// trace and statistics of the schedule returned on the host.  Calls on one
// device are serialised; each call synchronises its stream before returning.
#pragma once
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "ofx_desc.cuh"
#include "ofx_passx.cuh"
#include "../../include/optifax.h"

namespace ofx {

template <typename R>
struct XKernel {
    void (*fn)(const PulseX*, XTables<R>, KernelCfg);
    size_t smem;
    int threads, M, C;
    bool nee;
};

template <typename R, int M, int C, bool NEE>
XKernel<R> xkernel() {
    return XKernel<R>{&passx_kernel<R, M, C, NEE>, SmemX<R, M, C>::bytes, ShapeX<M, C>::T, M, C, NEE};
}

// W_N^e for e < N in FP64, rounded to R
template <typename R>
__global__ void passx_twiddles(typename Num<R>::cplx* out, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    double s, c;
    sincospi(-2.0 * (double)e / (double)n, &s, &c);
    out[e] = Num<R>::from(make_double2(c, s));
}

// How many clusters of a kernel the GPU holds at once (0 on an error)
template <typename R>
inline int xresident(const XKernel<R>& k) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)k.C, 1, 1);
    lc.blockDim = dim3((unsigned)k.threads, 1, 1);
    lc.dynamicSmemBytes = k.smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = k.C; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    lc.attrs = &attr;
    lc.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k.fn, &lc) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <typename R>
inline cudaError_t xattributes(const XKernel<R>& k) {
    cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    if (e == cudaSuccess && k.C > 8) e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// The kernel of n points for a call of B pulses.  The FP64 rate and the serial chain
// bound these kernels, so a pulse takes as many SMs as a cluster allows: 512 points per
// CTA up to 2^13 points, then n / 16 (one pulse, us per attempt, GB300, FP64 at 1024 and
// 512 points per CTA: 2^10 38 and 26, 2^12 48 and 30, 2^13 53 and 33; float-float at 2^13
// 19 and 16; measured before the absorber's factors were kept, now 24, 28, 30 and 12.5 at
// 512).  Several pulses on one schedule run at once: at 2^13 points the GPU holds 14 of
// them at 512 points per CTA and one more at 1024 (below, it holds as many at 512 as a
// call may have; above, there is one shape).
template <typename R>
inline const XKernel<R>* xchoose(const std::vector<XKernel<R>>& kernels, int n, int B, bool nee) {
    auto find = [&](int m) -> const XKernel<R>* {
        if (n / m > 16) m = n / 16;
        for (const auto& k : kernels)
            if (k.M == m && k.C == n / m && k.nee == nee) return &k;
        return nullptr;
    };
    const XKernel<R>* wide = find(512);
    if (n != 8192 || B == 1 || !wide) return wide;
    return xattributes(*wide) != cudaSuccess || B > xresident(*wide) ? find(1024) : wide;
}

// What a call reads back: the schedule's statistics and the shared schedule's words
struct XReport {
    optifax_pulse_stats stats;
    unsigned long long sync[4];
};

template <typename R>
struct XWork {
    int n_tab = 0;
    typename Num<R>::cplx* tab = nullptr;
    void* ztab = nullptr;
    size_t ztab_bytes = 0;
    PulseX* desc = nullptr;
    size_t desc_n = 0;
    int* trace = nullptr;
    size_t trace_n = 0;
    XReport* report = nullptr;
};

template <typename T>
inline int grow_dev(T** p, size_t* have, size_t need_bytes) {
    if (*p && *have >= need_bytes) return OPTIFAX_OK;
    if (*p) { cudaFree(*p); *p = nullptr; *have = 0; }
    if (cudaMalloc((void**)p, need_bytes) != cudaSuccess) return OPTIFAX_ERR_NO_MEMORY;
    *have = need_bytes;
    return OPTIFAX_OK;
}

template <typename R>
int passx_run(const std::vector<XKernel<R>>& kernels, XWork<R>& w, int n, int B, int S, const double* E_in,
              double* A_out, const double* alpha, const double* beta, const double* G, int g_per_pulse,
              double w0, double bdiffw0, double step_h, double dt, double max_err, double min_err, double sel,
              int variant, int32_t* trace_host, int32_t trace_cap, optifax_pulse_stats* stats_host,
              cudaStream_t st) {
    if (!is_pow2(n) || n < 512 || n > 65536 || B < 1 || S < 1 || !(sel >= 1.0) || !E_in || !A_out || !alpha ||
        !beta || !G || !(step_h > 0.0) || !(dt > 0.0) || !(w0 > 0.0) || (trace_host && trace_cap < 0))
        return OPTIFAX_ERR_INVALID_ARGUMENT;
    if (64LL * (S + 16) + 64 > 0x7fffffffLL) return OPTIFAX_ERR_INVALID_ARGUMENT;
    VariantCfg vc;
    if (variant == OPTIFAX_VARIANT_ODE23 || !variant_cfg(variant, &vc)) return OPTIFAX_ERR_INVALID_ARGUMENT;
    const XKernel<R>* ke = xchoose(kernels, n, B, vc.nee != 0);
    if (!ke) return OPTIFAX_ERR_UNSUPPORTED;
    const int C = ke->C;
    // one co-resident wave (cooperative launch), counted in the narrow shape
    const int narrow = n < 1024 || (std::is_same<R, ff>::value && n <= 4096) ? 512 : 1024;
    if (B > 1 && B * (n / narrow > 16 ? 16 : n / narrow) > 148) return OPTIFAX_ERR_UNSUPPORTED;

    int rc;
    using cplx = typename Num<R>::cplx;
    if (w.n_tab != n) {
        size_t have = w.tab ? sizeof(cplx) * (size_t)w.n_tab : 0;
        if ((rc = grow_dev(&w.tab, &have, sizeof(cplx) * (size_t)n))) { w.n_tab = 0; return rc; }
        passx_twiddles<R><<<(n + 255) / 256, 256, 0, st>>>(w.tab, n);
        if (cudaGetLastError() != cudaSuccess) { w.n_tab = 0; return OPTIFAX_ERR_CUDA; }
        w.n_tab = n;
    }
    const int zcap = S + 64;     // z-samples k + stepmod of a pass stay below S + stepmod's clamp
    if ((rc = grow_dev(&w.ztab, &w.ztab_bytes, sizeof(cplx) * (size_t)zcap * B))) return rc;
    size_t dn = w.desc_n * sizeof(PulseX);
    if ((rc = grow_dev(&w.desc, &dn, sizeof(PulseX) * (size_t)B))) return rc;
    w.desc_n = dn / sizeof(PulseX);
    const size_t tcap = trace_host ? (size_t)trace_cap : 0;
    size_t tn = w.trace_n * 3 * sizeof(int);
    if (tcap && (rc = grow_dev(&w.trace, &tn, 3 * sizeof(int) * tcap))) return rc;
    if (tcap) w.trace_n = tn / (3 * sizeof(int));
    size_t rb = w.report ? sizeof(XReport) : 0;
    if ((rc = grow_dev(&w.report, &rb, sizeof(XReport)))) return rc;

    std::vector<PulseX> d((size_t)B);
    int nchunks = (int)((double)S / sel);
    if (vc.guard && (double)nchunks * sel < (double)S) nchunks += 1;
    for (int b = 0; b < B; ++b) {
        PulseX& x = d[(size_t)b];
        memset(&x, 0, sizeof(x));
        x.E_in = reinterpret_cast<const double2*>(E_in) + (size_t)b * n;
        x.A_out = reinterpret_cast<double2*>(A_out) + (size_t)b * n;
        x.alpha = alpha;
        x.beta = beta;
        x.G = G + (g_per_pulse ? (size_t)b * S : 0);
        x.trace = (b == 0 && tcap) ? w.trace : nullptr;
        x.trace_cap = (b == 0) ? (int)tcap : 0;
        x.stats = (b == 0) ? &w.report->stats : nullptr;
        x.ztab = reinterpret_cast<cplx*>(w.ztab) + (size_t)b * zcap;
        x.zcap = zcap;
        x.tau_theta = turns_fixed((long double)w0 * (long double)dt);
        x.tau_z = turns_fixed((long double)bdiffw0 * (long double)step_h);
        x.w0 = w0; x.h = step_h; x.dt = dt;
        x.max_err = max_err; x.min_err = min_err; x.sel = sel;
        x.c_shock = 1.0 / (2.0 * dt * w0);
        x.N = n; x.S = S; x.nchunks = nchunks;
    }
    if (cudaMemcpyAsync(w.desc, d.data(), sizeof(PulseX) * (size_t)B, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(w.report, 0, sizeof(XReport), st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    if (xattributes(*ke) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    KernelCfg cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.time_mode = vc.time_mode;
    cfg.abc_mode = vc.abc_mode;
    cfg.guard = vc.guard;
    cfg.shared_sched = B > 1 ? 1 : 0;
    cfg.max_attempts_mul = 64;
    cfg.grid_sync = w.report->sync;
    cfg.clusters = B;
    cfg.wait = kWait;
    XTables<R> tabs;
    tabs.wn = w.tab;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(B * C), 1, 1);
    lc.blockDim = dim3((unsigned)ke->threads, 1, 1);
    lc.dynamicSmemBytes = ke->smem;
    lc.stream = st;
    cudaLaunchAttribute attrs[2];
    int na = 0;
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = C; attrs[na].val.clusterDim.y = 1; attrs[na].val.clusterDim.z = 1;
    ++na;
    if (B > 1) {
        attrs[na].id = cudaLaunchAttributeCooperative;
        attrs[na].val.cooperative = 1;
        ++na;
    }
    lc.attrs = attrs;
    lc.numAttrs = na;
    const PulseX* dd = w.desc;
    if (cudaLaunchKernelEx(&lc, ke->fn, dd, tabs, cfg) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    XReport report;
    if (cudaMemcpyAsync(&report, w.report, sizeof(report), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return OPTIFAX_ERR_CUDA;
    const optifax_pulse_stats& hs = report.stats;
    if (tcap) {
        const size_t nt = (size_t)(hs.attempts < trace_cap ? hs.attempts : trace_cap);
        if (nt && cudaMemcpy(trace_host, w.trace, 3 * sizeof(int) * nt, cudaMemcpyDeviceToHost) != cudaSuccess)
            return OPTIFAX_ERR_CUDA;
    }
    if (stats_host) *stats_host = hs;
    // a wait of this or another pulse of the schedule ran out: its field is NaN
    return (hs.status & OPTIFAX_PULSE_TIMEOUT) || report.sync[3] ? OPTIFAX_ERR_CUDA : OPTIFAX_OK;
}

}  // namespace ofx
