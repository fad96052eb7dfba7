// The bounded waits of the crystal-pass kernels, made to run out by what nothing sends: built
// and driven by test_waits_gpu.py.
#include <cstdlib>
#include <vector>

#include "ofx_kernels.cuh"
#include "ofx_passx.cuh"

using namespace ofx;

namespace {

template <typename T>
struct Dev {
    T* p = nullptr;
    explicit Dev(size_t n) { cudaMalloc(&p, n * sizeof(T)); cudaMemset(p, 0, n * sizeof(T)); }
    Dev(const std::vector<T>& v) : Dev(v.size()) { cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice); }
    ~Dev() { cudaFree(p); }
};

template <typename K, typename... A>
int launch(K k, int clusters, int C, int threads, size_t smem, A... a) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 1;
    if (C > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(clusters * C);
    lc.blockDim = dim3(threads);
    lc.dynamicSmemBytes = smem;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    if (cudaLaunchKernelEx(&lc, k, a...) != cudaSuccess) return 2;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 3;
}

KernelCfg config(int expected, int wait, unsigned long long* sync) {
    KernelCfg c = {};
    c.shared_sched = 1;
    c.max_attempts_mul = 64;
    c.grid_sync = sync;
    c.clusters = expected;
    c.wait = wait;
    return c;
}

constexpr int kS = 64;

// Zero fields on a shared schedule of `clusters` that expects `expected`
template <int M, int C, int METHOD>
int run_pass(int clusters, int expected, int wait, int* status, float* out, int* flag) {
    constexpr int N = M * C;
    std::vector<Twiddle> one(M, Twiddle{1.f, 0.f, 0.f, 0.f});
    Dev<Twiddle> tab(one);
    Dev<float2> E(N), A((size_t)N * clusters);
    Dev<float> alpha(std::vector<float>(N, 1.f)), beta(N), G(kS);
    Dev<optifax_pulse_stats> st(clusters);
    Dev<unsigned long long> sync(4);
    std::vector<PulseDev> d(clusters);
    for (int i = 0; i < clusters; ++i) {
        d[i] = PulseDev{};
        d[i].E_in = E.p; d[i].A_out = A.p + (size_t)i * N; d[i].alpha = alpha.p; d[i].beta = beta.p; d[i].G = G.p;
        d[i].stats = st.p + i;
        d[i].w0 = 1.f; d[i].h = 1e-7f; d[i].max_err = 0.05f; d[i].min_err = 0.0025f; d[i].sel = kS;
        d[i].N = N; d[i].S = kS; d[i].nchunks = 1;
    }
    Dev<PulseDev> desc(d);
    const FftTables tabs{tab.p, tab.p};
    const int rc = launch(&pass_kernel<M, C, METHOD>, clusters, C, M / kPoints<M>, Smem<M, METHOD, C>::bytes,
                          (const PulseDev*)desc.p, tabs, config(expected, wait, sync.p));
    if (rc) return rc;
    std::vector<optifax_pulse_stats> hs(clusters);
    unsigned long long hw[4];
    cudaMemcpy(hs.data(), st.p, sizeof(optifax_pulse_stats) * clusters, cudaMemcpyDeviceToHost);
    cudaMemcpy(hw, sync.p, sizeof(hw), cudaMemcpyDeviceToHost);
    cudaMemcpy(out, A.p, sizeof(float2) * (size_t)N * clusters, cudaMemcpyDeviceToHost);
    for (int i = 0; i < clusters; ++i) status[i] = hs[i].status;
    *flag = (int)hw[3];
    return 0;
}

template <int M, int C>
int run_wide(int clusters, int expected, int wait, int* status, float* out, int* flag) {
    constexpr int N = M * C;
    Dev<double2> wn(std::vector<double2>(N, make_double2(1.0, 0.0))), E(N), A((size_t)N * clusters), z(kS + 64);
    Dev<double> alpha(std::vector<double>(N, 1.0)), beta(N), G(kS);
    Dev<optifax_pulse_stats> st(clusters);
    Dev<unsigned long long> sync(4);
    std::vector<PulseX> d(clusters);
    for (int i = 0; i < clusters; ++i) {
        d[i] = PulseX{};
        d[i].E_in = E.p; d[i].A_out = A.p + (size_t)i * N; d[i].alpha = alpha.p; d[i].beta = beta.p; d[i].G = G.p;
        d[i].stats = st.p + i; d[i].ztab = z.p; d[i].zcap = kS + 64;
        d[i].w0 = 1.0; d[i].h = 1e-7; d[i].dt = 1e-15; d[i].max_err = 0.05; d[i].min_err = 0.0025; d[i].sel = kS;
        d[i].N = N; d[i].S = kS; d[i].nchunks = 1;
    }
    Dev<PulseX> desc(d);
    const XTables<double> tabs{wn.p};
    const int rc = launch(&passx_kernel<double, M, C, false>, clusters, C, ShapeX<M, C>::T, SmemX<double, M, C>::bytes,
                          (const PulseX*)desc.p, tabs, config(expected, wait, sync.p));
    if (rc) return rc;
    std::vector<optifax_pulse_stats> hs(clusters);
    std::vector<double> ho((size_t)2 * N * clusters);
    unsigned long long hw[4];
    cudaMemcpy(hs.data(), st.p, sizeof(optifax_pulse_stats) * clusters, cudaMemcpyDeviceToHost);
    cudaMemcpy(hw, sync.p, sizeof(hw), cudaMemcpyDeviceToHost);
    cudaMemcpy(ho.data(), A.p, sizeof(double) * ho.size(), cudaMemcpyDeviceToHost);
    for (int i = 0; i < clusters; ++i) status[i] = hs[i].status;
    for (size_t i = 0; i < ho.size(); ++i) out[i] = (float)ho[i];
    *flag = (int)hw[3];
    return 0;
}

// One attempt's flags in a cluster of two.  what = 0: both send; 1: CTA 1 sends nothing and
// stays; 2: CTA 1 knows of a wait that ran out.  Then CTA 1 (or, in 0, both) takes the
// barrier of a rejected step, and a CTA that combine_flags ended its last one.
// out[rank][thread] = flags, or kDead; 64 added where the reject barrier met the other's last.
constexpr int kT = 128, kNW = kT / 32;
__global__ void __cluster_dims__(2) flag_kernel(int what, KernelCfg cfg, int* out) {
    __shared__ __align__(16) int red[2 * kNW + 2 * 16 + 8];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ unsigned long long last[3];
    int* dead = red + 2 * kNW + 2 * 16;
    const int t = threadIdx.x, c = (int)cg::this_cluster().block_rank();
    const uint32_t bar = smem_u32(&bar_s);
    if (t < 2 * kNW + 2 * 16 + 8) red[t] = 0;
    __syncthreads();
    if (t == 0) {
        if (what == 2 && c == 1) dead[0] = 1;
        bar_init(bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_arm(bar, 4);
    }
    cg::this_cluster().sync();
    int f = 0;
    if (!(what == 1 && c == 1))
        f = combine_flags<kNW, 2>(t == 5 ? 1 + c : 0, red, bar, 0, 4, dead, last, 0, t, c, cfg);
    __shared__ float2 nowhere[2];
    bool gone = false;
    if (!(f & kDead)) {
        count_bar(dead, t);
        cg::this_cluster().sync();
        gone = peer_gone(dead);
    }
    if (!last_word<2>(dead)) cg::this_cluster().sync();
    end_lost<1, 2, float2>(dead, nowhere, nullptr, cfg);
    out[c * kT + t] = f | (gone ? 64 : 0) | ((dead[0] | dead[kTold]) ? 128 : 0);
}

}  // namespace

extern "C" int wait_pass(int kind, int clusters, int expected, int wait, int* status, float* out, int* flag) {
    switch (kind) {
        case 0: return run_pass<512, 1, OPTIFAX_HEUN>(clusters, expected, wait, status, out, flag);
        case 1: return run_pass<512, 2, OPTIFAX_HEUN>(clusters, expected, wait, status, out, flag);
        case 2: return run_pass<512, 2, OPTIFAX_RK23>(clusters, expected, wait, status, out, flag);
        case 3: return run_pass<1024, 16, OPTIFAX_HEUN>(clusters, expected, wait, status, out, flag);
        default: return run_wide<512, 2>(clusters, expected, wait, status, out, flag);
    }
}

extern "C" int wait_flags(int what, int wait, int* out) {
    Dev<int> o(2 * kT);
    KernelCfg cfg = {};
    cfg.wait = wait;
    flag_kernel<<<2, kT>>>(what, cfg, o.p);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return 1;
    return cudaMemcpy(out, o.p, sizeof(int) * 2 * kT, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 2;
}
