// ofx_api.cu -- C ABI (include/optifax.h): context, twiddle tables,
// descriptor staging, validation and launch of the crystal-pass kernels.
//
// Replaces the MEX gateway mexFunction (toolbox/lib/MEXlib/src/OPO_mex_BATCH.cpp:19-141)
// and the host driver OPO_TEST_CUDA (OPO_CUDA_BATCH_XTAL.cu:373-525,
// ode23/OPO_CUDA_ODE23.cu:375-557): instead of ~10 launches, two cuFFT calls
// and two device synchronisations per step, one launch runs every step of
// every pulse.
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "ofx_kernels.cuh"
#include "ofx_desc.cuh"
#include "ofx_gnlse.cuh"
#include "../../include/optifax.h"

using namespace ofx;

struct optifax_context {
    int device = 0;
    std::map<int, Twiddle*> tw;          // N -> W_N^i, i < 64 (cluster exchange)
    std::map<int, Twiddle*> quadtw;      // M -> W_M^y, y < M/4 (cluster exchange)
    PulseDev* d_desc = nullptr;
    size_t desc_cap = 0;
    float2* d_xs = nullptr;              // cavities' trip-output scratch
    size_t xs_cap = 0;                   // in complex values
    std::vector<cudaStream_t> side;      // streams for concurrent launch groups
    std::vector<cudaEvent_t> ev;         // fork/join events
    unsigned long long* d_grid_sync = nullptr;   // shared schedules: 4 words
    ofx::GnlseDev* d_gnlse_desc = nullptr;   // GNLSE: descriptors and stage scratch
    size_t gnlse_desc_cap = 0;
    float2* d_gnlse_k = nullptr;
    size_t gnlse_k_cap = 0;                  // complex values
    std::map<const void*, int> resident;     // kernel -> clusters that fit the GPU at once
    int cta_points = 0;                      // of calls and pulses without a choice of their own; 0: the rule's
    cudaEvent_t done_ev = nullptr;           // end of the last call's work on the GPU
    bool done_pending = false;               // done_ev has been recorded
    std::string last_error;
};

namespace {

// out[e] = W_n^e = exp(-2 pi i e / n) for e < count, rounded to FP32, with
// d = 1/|w|^2 - 1 in FP64.  The cluster exchange's tables: the quarter period of
// W_M (count M/4) and W_N^i for i < 64 (also the source of the crystal pass's FFT tables).
__global__ void twiddle_kernel(Twiddle* out, int n, int count) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= count) return;
    double s, c;
    sincospi(-2.0 * (double)e / (double)n, &s, &c);
    float cf = (float)c, sf = (float)s;
    double m2 = (double)cf * (double)cf + (double)sf * (double)sf;
    Twiddle w;
    w.c = cf; w.s = sf; w.d = (float)(1.0 / m2 - 1.0); w.pad = 0.f;
    out[e] = w;
}

int fail(optifax_context* h, int code, const std::string& msg) {
    if (h) h->last_error = msg;
    return code;
}

int cuda_fail(optifax_context* h, cudaError_t e, const char* what) {
    return fail(h, OPTIFAX_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// Every call stages its descriptors into, and runs on, device scratch owned by the
// handle, so its work waits for the previous call's (done_ev).  On the previous
// call's own stream the wait adds nothing to stream order; it is made on every
// stream because a stream handle's value can be reused after the stream is destroyed.
int order_after_previous(optifax_context* h, cudaStream_t st) {
    if (!h->done_pending) return OPTIFAX_OK;
    cudaError_t e = cudaStreamWaitEvent(st, h->done_ev, 0);
    return e == cudaSuccess ? OPTIFAX_OK : cuda_fail(h, e, "cudaStreamWaitEvent(previous call)");
}

int mark_done(optifax_context* h, cudaStream_t st) {
    cudaError_t e = cudaEventRecord(h->done_ev, st);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaEventRecord(end of call)");
    h->done_pending = true;
    return OPTIFAX_OK;
}

// Grow a handle-owned scratch buffer in stream order: the old buffer goes back
// with cudaFreeAsync once the previous call's work is done (the stream waits on
// done_ev first), the new one comes from cudaMallocAsync on the same stream, so
// no other work on the device is waited for.
int grow_scratch(optifax_context* h, void** buf, size_t* cap_bytes, size_t need_bytes, cudaStream_t st,
                 const char* what) {
    if (*buf && need_bytes <= *cap_bytes) return OPTIFAX_OK;
    int rc = order_after_previous(h, st);
    if (rc) return rc;
    if (*buf) {
        cudaError_t e = cudaFreeAsync(*buf, st);
        if (e != cudaSuccess) return cuda_fail(h, e, what);
        *buf = nullptr;
        *cap_bytes = 0;
    }
    cudaError_t e = cudaMallocAsync(buf, need_bytes, st);
    if (e != cudaSuccess) { *buf = nullptr; return cuda_fail(h, e, what); }
    *cap_bytes = need_bytes;
    return OPTIFAX_OK;
}

// W_n^e for e < count, built once per (n, count) map and kept for the context
const Twiddle* get_table(optifax_context* h, std::map<int, Twiddle*>& cache, int n, int count,
                         cudaStream_t st, int* rc) {
    auto it = cache.find(n);
    if (it != cache.end()) return it->second;
    Twiddle* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(Twiddle) * (size_t)count);
    if (e != cudaSuccess) { *rc = cuda_fail(h, e, "cudaMalloc(twiddles)"); return nullptr; }
    twiddle_kernel<<<(count + 255) / 256, 256, 0, st>>>(d, n, count);
    e = cudaGetLastError();
    if (e != cudaSuccess) { cudaFree(d); *rc = cuda_fail(h, e, "twiddle_kernel"); return nullptr; }
    // tables are shared by every stream of the context: finish building them now
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { cudaFree(d); *rc = cuda_fail(h, e, "twiddle_kernel sync"); return nullptr; }
    cache[n] = d;
    return d;
}

const std::vector<KernelEntry>& kernel_table() {
    static const std::vector<KernelEntry> tbl = [] {
        std::vector<KernelEntry> v;
        register_kernels_heun_large(v);
        register_kernels_heun_small(v);
        register_kernels_rk23(v);
        register_kernels_heun_nee(v);
        return v;
    }();
    return tbl;
}

const KernelEntry* find_kernel(int M, int C, int method) {
    for (const auto& k : kernel_table())
        if (k.M == M && k.C == C && k.method == method) return &k;
    return nullptr;
}

struct Group {
    int M, C;
    std::vector<PulseDev> d;
};

// Kernel attributes (dynamic shared memory, 16-CTA clusters): not stream work, so set
// before the launches (and outside any capture).
cudaError_t set_attributes(const KernelEntry& ke) {
    cudaError_t e = cudaFuncSetAttribute(ke.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ke.smem);
    if (e == cudaSuccess && ke.C > 8) e = cudaFuncSetAttribute(ke.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// How many clusters of a kernel the GPU holds at once
int resident_clusters(optifax_context* h, const KernelEntry& ke) {
    auto it = h->resident.find((const void*)ke.fn);
    if (it != h->resident.end()) return it->second;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)ke.C, 1, 1);
    lc.blockDim = dim3((unsigned)ke.threads, 1, 1);
    lc.dynamicSmemBytes = ke.smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ke.C; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    lc.attrs = &attr;
    lc.numAttrs = 1;
    int n = 0;
    if (set_attributes(ke) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, ke.fn, &lc) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    h->resident[(const void*)ke.fn] = n;
    return n;
}

// Points per CTA of a grid of N points that carries no choice of the caller, by spread:
//   0  the shortest time per attempt of one pulse
//   1  half the CTAs; at 2048 points one CTA (two of 1024 points are slower and twice the SMs)
//   2  4096 points per CTA (one CTA up to 4096 points): the least SM time per attempt
// One pulse, us per attempt (GB300, 2 W, 30 um poling), at spread 2 -> 1 -> 0:
//            2048 (1024 x 2)       4096          8192              16384             32768
//   Heun  3.8 (4.0)  -> 3.0   6.5 4.2 3.3   9.1 5.9 4.2   9.6 5.7 4.9    9.9  9.9 6.8
//   RK23  4.8 (4.6)  -> 3.5   7.6  -  3.6  10.3 6.6 4.5  10.8 8.9 5.2
//   NEE   3.7 (3.9)  -> 2.9   6.4  -  3.2   9.1 5.9 4.2   9.6 5.7 4.7
// SM time per attempt goes the other way (4096: 6.5, 17, 26 SM us), so the wider
// spreads serve calls that leave SMs idle otherwise.
int spread_points(int N, int spread) {
    const int narrow = N <= 4096 ? N : 4096;
    if (N <= 1024 || N > 32768 || spread >= 2) return narrow;
    const int wide = N <= 4096 ? 512 : N == 32768 ? 2048 : 1024;
    return spread == 0 ? wide : (N > 2048 && 2 * wide < narrow ? 2 * wide : narrow);
}

// One pulse of a call before its group is known
struct Placed {
    PulseDev d;
    int want;        // points per CTA asked for, 0: the rule's choice
};

int no_kernel(optifax_context* h, int M, int C) {
    return fail(h, OPTIFAX_ERR_UNSUPPORTED,
                "no kernel for cta_points=" + std::to_string(M) + " cluster=" + std::to_string(C));
}

// Handles alive on each device.  The calls of one handle do not overlap, so this many calls
// at most run there at once.
std::atomic<int> g_alive[64];

// Groups the pulses by (cta_points, cluster).  Pulses without a choice of the caller
// take the widest spread at which every cluster of this call, and of one such call on every
// other handle of the device, is resident at once (each kernel's clusters as a share of
// what the GPU holds of it), else the narrow one.  Without regard to the other handles,
// 150 handles with a pulse of 16384 points each took 47.6 ms on 16 CTAs a pulse, and 21.3 ms
// on 4 as now; 32 handles 10.9 and 4.5; 150 of 4096 points 11.8 (8 CTAs) and 8.5.
int group_pulses(optifax_context* h, std::vector<Placed>& pulses, int method, std::vector<Group>* gv) {
    const int calls = std::max(1, h->device < 64 ? g_alive[h->device].load(std::memory_order_relaxed) : 1);
    for (Placed& p : pulses)
        if (p.want == 0) p.want = h->cta_points;
    auto points = [&](const Placed& p, int spread) {
        const int narrow = p.d.N <= 4096 ? p.d.N : 4096;
        if (p.want > 0) return p.want < p.d.N ? p.want : p.d.N;
        const int M = spread_points(p.d.N, spread);
        // sizes without a kernel at 4096 points per CTA stay refused
        return find_kernel(narrow, p.d.N / narrow, method) && find_kernel(M, p.d.N / M, method) ? M : narrow;
    };
    for (const Placed& p : pulses) {
        const int M = points(p, 2), C = p.d.N / M;
        if (C > 16) return fail(h, OPTIFAX_ERR_UNSUPPORTED, "n_points / cta_points exceeds 16");
        const KernelEntry* ke = find_kernel(M, C, method);
        if (!ke || (p.want > 0 && ke->rule_only)) return no_kernel(h, M, C);
    }
    int spread = 0;
    for (; spread < 2; ++spread) {
        std::map<std::pair<int, int>, int> count;
        for (const Placed& p : pulses) {
            const int M = points(p, spread);
            ++count[{M, p.d.N / M}];
        }
        double share = 0.0;
        for (const auto& g : count) {
            const KernelEntry* ke = find_kernel(g.first.first, g.first.second, method);
            const int n = ke ? resident_clusters(h, *ke) : 0;
            share += n > 0 ? (double)g.second / n : 2.0;
        }
        if (share * calls <= 1.0) break;
    }
    std::map<std::pair<int, int>, std::vector<PulseDev>> groups;
    for (const Placed& p : pulses) {
        const int M = points(p, spread);
        groups[{M, p.d.N / M}].push_back(p.d);
    }
    gv->clear();
    for (auto& g : groups) gv->push_back(Group{g.first.first, g.first.second, std::move(g.second)});
    return OPTIFAX_OK;
}

double pulse_cost(const PulseDev& d) {
    return (double)d.N * std::log2((double)d.N) * (double)d.S;
}

int ensure_sync_objects(optifax_context* h, size_t n_streams) {
    while (h->side.size() < n_streams) {
        cudaStream_t s_;
        cudaError_t e = cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaStreamCreate");
        h->side.push_back(s_);
    }
    while (h->ev.size() < n_streams + 1) {
        cudaEvent_t e_;
        cudaError_t e = cudaEventCreateWithFlags(&e_, cudaEventDisableTiming);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaEventCreate");
        h->ev.push_back(e_);
    }
    return OPTIFAX_OK;
}

// Order the groups for launch (longest work first within a group; groups in order
// of their longest pulse, longest first: the block scheduler serves earlier
// launches first, so the critical path starts at once and large clusters find
// whole GPCs free only at the start) and return the scratch that their cavities need
// (complex values: the trip's crystal output of each).
size_t order_groups(std::vector<Group>& groups) {
    for (auto& g : groups) {
        std::stable_sort(g.d.begin(), g.d.end(),
                         [](const PulseDev& x, const PulseDev& y) { return pulse_cost(x) > pulse_cost(y); });
    }
    auto group_key = [](const Group& g) { return g.d.empty() ? 0.0 : pulse_cost(g.d.front()); };
    std::stable_sort(groups.begin(), groups.end(),
                     [&](const Group& x, const Group& y) { return group_key(x) > group_key(y); });
    size_t need_xs = 0;
    for (auto& g : groups)
        for (const auto& d : g.d)
            if (d.fb) need_xs += (size_t)g.M * g.C;
    return need_xs;
}

// Descriptors in launch order with their cavity scratch carved from xs.
std::vector<PulseDev> place_descriptors(std::vector<Group>& groups, float2* xs) {
    std::vector<PulseDev> all;
    size_t xoff = 0;
    for (auto& g : groups)
        for (auto& d : g.d) {
            if (d.fb) { d.xs = xs + xoff; xoff += (size_t)g.M * g.C; }
            all.push_back(d);
        }
    return all;
}

// The FFT tables of every group, built (once per context) before any launch:
// building one synchronises the stream, which must not happen between launches.
int group_tables(optifax_context* h, const std::vector<Group>& groups, cudaStream_t st, std::vector<FftTables>* tabv) {
    int rc = OPTIFAX_OK;
    tabv->assign(groups.size(), FftTables{});
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        const int M = groups[gi].M;
        (*tabv)[gi].quad = get_table(h, h->quadtw, M, M / 4, st, &rc);       // quarter period of W_M
        if (!(*tabv)[gi].quad) return rc;
        (*tabv)[gi].low = get_table(h, h->tw, M * groups[gi].C, 64, st, &rc);  // W_N^i, i < 64
        if (!(*tabv)[gi].low) return rc;
    }
    return rc;
}

int group_attributes(optifax_context* h, const std::vector<Group>& groups, int method, const VariantCfg& vc) {
    for (const auto& g : groups) {
        const KernelEntry* ke = find_kernel(g.M, g.C, vc.nee ? kHeunNee : method);
        if (!ke) return no_kernel(h, g.M, g.C);
        cudaError_t e = set_attributes(*ke);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaFuncSetAttribute");
    }
    return OPTIFAX_OK;
}

// One grid per (cta_points, cluster) group; groups after the first run on side
// streams forked from and joined back into `st`, so the block scheduler
// interleaves them: CTAs of a long group fill SMs as short ones end.
int enqueue_groups(optifax_context* h, const std::vector<Group>& groups, int method, const VariantCfg& vc,
                   bool shared, const PulseDev* d_desc, const std::vector<FftTables>& tabv, unsigned long long* grid_sync,
                   cudaStream_t st, const std::vector<cudaStream_t>& side, const std::vector<cudaEvent_t>& ev) {
    cudaError_t e;
    if (groups.size() > 1) {
        e = cudaEventRecord(ev[0], st);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaEventRecord");
    }
    size_t off = 0;
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        const Group& g = groups[gi];
        const int M = g.M, C = g.C;
        const KernelEntry* ke = find_kernel(M, C, vc.nee ? kHeunNee : method);
        if (!ke) return no_kernel(h, M, C);
        const FftTables tabs = tabv[gi];
        KernelCfg cfg;
        cfg.time_mode = vc.time_mode;
        cfg.abc_mode = vc.abc_mode;
        cfg.guard = vc.guard;
        cfg.shared_sched = shared ? 1 : 0;
        cfg.max_attempts_mul = 64;
        cfg.grid_sync = grid_sync;
        cfg.clusters = (int)g.d.size();
        cfg.wait = kWait;
        cudaStream_t ls = st;
        if (gi > 0) {
            ls = side[gi - 1];
            e = cudaStreamWaitEvent(ls, ev[0], 0);
            if (e != cudaSuccess) return cuda_fail(h, e, "cudaStreamWaitEvent(fork)");
        }
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)(g.d.size() * C), 1, 1);
        lc.blockDim = dim3((unsigned)ke->threads, 1, 1);
        lc.dynamicSmemBytes = ke->smem;
        lc.stream = ls;
        cudaLaunchAttribute attrs[2];
        int na = 0;
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = C; attrs[na].val.clusterDim.y = 1; attrs[na].val.clusterDim.z = 1;
        ++na;
        if (shared) {
            attrs[na].id = cudaLaunchAttributeCooperative;
            attrs[na].val.cooperative = 1;
            ++na;
        }
        lc.attrs = attrs;
        lc.numAttrs = na;
        const PulseDev* dd = d_desc + off;
        e = cudaLaunchKernelEx(&lc, ke->fn, dd, tabs, cfg);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaLaunchKernelEx(pass_kernel)");
        if (gi > 0) {
            e = cudaEventRecord(ev[gi], ls);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(st, ev[gi], 0);
            if (e != cudaSuccess) return cuda_fail(h, e, "join side stream");
        }
        off += g.d.size();
    }
    return OPTIFAX_OK;
}

// Stage every group's descriptors into the handle's scratch and launch the groups.
int launch_groups(optifax_context* h, std::vector<Group>& groups, int method, const VariantCfg& vc,
                  bool shared, cudaStream_t st) {
    const size_t need_xs = order_groups(groups);
    if (need_xs > h->xs_cap) {
        size_t cap = h->xs_cap * sizeof(float2);
        int grc = grow_scratch(h, (void**)&h->d_xs, &cap, need_xs * sizeof(float2), st,
                               "cudaMallocAsync(cavity scratch)");
        h->xs_cap = cap / sizeof(float2);
        if (grc) return grc;
    }
    std::vector<PulseDev> all = place_descriptors(groups, h->d_xs);
    size_t nb = all.size() * sizeof(PulseDev);
    if (nb > h->desc_cap) {
        int grc = grow_scratch(h, (void**)&h->d_desc, &h->desc_cap, nb < 4096 ? 4096 : nb * 2, st,
                               "cudaMallocAsync(descriptors)");
        if (grc) return grc;
    }
    int rc = order_after_previous(h, st);
    if (rc) return rc;
    cudaError_t e = cudaMemcpyAsync(h->d_desc, all.data(), nb, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaMemcpyAsync(descriptors)");
    if (shared) {
        e = cudaMemsetAsync(h->d_grid_sync, 0, 4 * sizeof(unsigned long long), st);
        if (e != cudaSuccess) return cuda_fail(h, e, "cudaMemsetAsync(grid sync)");
    }
    rc = ensure_sync_objects(h, groups.size());
    if (rc) return rc;
    std::vector<FftTables> tabv;
    rc = group_tables(h, groups, st, &tabv);
    if (rc) return rc;
    rc = group_attributes(h, groups, method, vc);
    if (rc) return rc;
    rc = enqueue_groups(h, groups, method, vc, shared, h->d_desc, tabv, h->d_grid_sync, st, h->side, h->ev);
    if (rc) return rc;
    return mark_done(h, st);
}

int fill_desc(optifax_context* h, const optifax_pulse& in, const VariantCfg& vc, PulseDev* d,
              optifax_pulse_stats* stats) {
    std::string why;
    int rc = fill_pulse_desc(in, vc, d, stats, &why);
    return rc ? fail(h, rc, why) : OPTIFAX_OK;
}

}  // namespace

extern "C" {

int optifax_create(optifax_handle* out, int device) {
    if (!out) return OPTIFAX_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n <= 0) return OPTIFAX_ERR_CUDA;
    if (device < 0 || device >= n) return OPTIFAX_ERR_INVALID_ARGUMENT;
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return OPTIFAX_ERR_CUDA;
    optifax_context* h = new (std::nothrow) optifax_context();
    if (!h) return OPTIFAX_ERR_NO_MEMORY;
    h->device = device;
    e = cudaMalloc(&h->d_grid_sync, 4 * sizeof(unsigned long long));
    if (e != cudaSuccess) { delete h; return OPTIFAX_ERR_CUDA; }
    e = cudaEventCreateWithFlags(&h->done_ev, cudaEventDisableTiming);
    if (e != cudaSuccess) { cudaFree(h->d_grid_sync); delete h; return OPTIFAX_ERR_CUDA; }
    if (device < 64) ++g_alive[device];
    *out = h;
    return OPTIFAX_OK;
}

int optifax_set_cta_points(optifax_handle h, int32_t cta_points) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    if (cta_points != 0 && (!is_pow2(cta_points) || cta_points < 512 || cta_points > 4096))
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "cta_points must be 0 or a power of two in [512, 4096]");
    h->cta_points = cta_points;
    return OPTIFAX_OK;
}

int optifax_destroy(optifax_handle h) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    cudaSetDevice(h->device);
    cudaDeviceSynchronize();
    for (auto& kv : h->tw) cudaFree(kv.second);
    for (auto& kv : h->quadtw) cudaFree(kv.second);
    if (h->d_desc) cudaFree(h->d_desc);
    if (h->d_grid_sync) cudaFree(h->d_grid_sync);
    if (h->d_xs) cudaFree(h->d_xs);
    if (h->d_gnlse_desc) cudaFree(h->d_gnlse_desc);
    if (h->d_gnlse_k) cudaFree(h->d_gnlse_k);
    for (auto s_ : h->side) cudaStreamDestroy(s_);
    for (auto e_ : h->ev) cudaEventDestroy(e_);
    if (h->done_ev) cudaEventDestroy(h->done_ev);
    if (h->device < 64) --g_alive[h->device];
    delete h;
    return OPTIFAX_OK;
}

const char* optifax_status_string(int status) {
    switch (status) {
        case OPTIFAX_OK: return "ok";
        case OPTIFAX_ERR_INVALID_ARGUMENT: return "invalid argument";
        case OPTIFAX_ERR_UNSUPPORTED: return "unsupported configuration";
        case OPTIFAX_ERR_CUDA: return "CUDA error";
        case OPTIFAX_ERR_NO_MEMORY: return "out of memory";
        case OPTIFAX_ERR_NULL_HANDLE: return "null handle";
        default: return "unknown status";
    }
}

const char* optifax_last_error(optifax_handle h) {
    return h ? h->last_error.c_str() : "null handle";
}

}  // extern "C"

namespace {

// Validation and grouping by (cta_points, cluster) shared by optifax_propagate and
// optifax_propagate_graph.
int propagate_groups(optifax_handle h, const optifax_pulse* pulses, int32_t n_pulses, int32_t method,
                     int32_t variant, int32_t cta_points, optifax_pulse_stats* stats, VariantCfg* vc,
                     std::vector<Group>* gv) {
    if (!pulses || n_pulses < 1) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "no pulses");
    if (method != OPTIFAX_HEUN && method != OPTIFAX_RK23)
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "unknown method");
    if (!variant_cfg(variant, vc)) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "unknown variant");
    if (vc->nee && method != OPTIFAX_HEUN)
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "the NEE variant is a Heun schedule (NEE_CPU.m)");
    if (cta_points != 0 && (!is_pow2(cta_points) || cta_points < 512 || cta_points > 4096))
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "cta_points must be 0 or a power of two in [512, 4096]");
    std::vector<Placed> placed((size_t)n_pulses);
    for (int i = 0; i < n_pulses; ++i) {
        int rc = fill_desc(h, pulses[i], *vc, &placed[i].d, stats ? stats + i : nullptr);
        if (rc) return rc;
        int want = pulses[i].cta_points > 0 ? pulses[i].cta_points : cta_points;
        if (want != 0 && (!is_pow2(want) || want < 512 || want > 4096))
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "pulse cta_points must be 0 or a power of two in [512, 4096]");
        placed[i].want = want;
    }
    return group_pulses(h, placed, vc->nee ? kHeunNee : method, gv);
}

}  // namespace

struct optifax_graph_s {
    int device = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    PulseDev* d_desc = nullptr;
    int kernels = 0;
};

extern "C" {

int optifax_propagate(optifax_handle h, const optifax_pulse* pulses, int32_t n_pulses,
                      int32_t method, int32_t variant, int32_t cta_points,
                      optifax_pulse_stats* stats, void* stream) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaSetDevice");
    VariantCfg vc;
    std::vector<Group> gv;
    int rc = propagate_groups(h, pulses, n_pulses, method, variant, cta_points, stats, &vc, &gv);
    if (rc) return rc;
    return launch_groups(h, gv, method, vc, false, (cudaStream_t)stream);
}

int optifax_graph_destroy(optifax_graph g) {
    if (!g) return OPTIFAX_ERR_INVALID_ARGUMENT;
    cudaSetDevice(g->device);
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    if (g->d_desc) cudaFree(g->d_desc);       // synchronises with any launch still running
    delete g;
    return OPTIFAX_OK;
}

int optifax_propagate_graph(optifax_handle h, const optifax_pulse* pulses, int32_t n_pulses,
                            int32_t method, int32_t variant, int32_t cta_points,
                            optifax_pulse_stats* stats, optifax_graph* out) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    if (!out) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "no output graph");
    *out = nullptr;
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaSetDevice");
    VariantCfg vc;
    std::vector<Group> gv;
    int rc = propagate_groups(h, pulses, n_pulses, method, variant, cta_points, stats, &vc, &gv);
    if (rc) return rc;
    optifax_graph g = new (std::nothrow) optifax_graph_s();
    if (!g) return fail(h, OPTIFAX_ERR_NO_MEMORY, "graph object");
    g->device = h->device;
    // the graph owns its descriptors: later calls on the handle neither move nor
    // overwrite them (passes without a cavity need no scratch)
    order_groups(gv);
    std::vector<PulseDev> all;
    cudaStream_t s0 = nullptr;
    std::vector<cudaStream_t> side;
    std::vector<cudaEvent_t> ev;
    std::vector<FftTables> tabv;
    auto cleanup = [&](int code) {
        for (auto s_ : side) cudaStreamDestroy(s_);
        for (auto e_ : ev) cudaEventDestroy(e_);
        if (s0) cudaStreamDestroy(s0);
        if (code) optifax_graph_destroy(g);
        return code;
    };
    all = place_descriptors(gv, nullptr);
    if ((e = cudaMalloc(&g->d_desc, all.size() * sizeof(PulseDev))) != cudaSuccess)
        return cleanup(cuda_fail(h, e, "cudaMalloc(graph descriptors)"));
    if ((e = cudaMemcpy(g->d_desc, all.data(), all.size() * sizeof(PulseDev), cudaMemcpyHostToDevice)) != cudaSuccess)
        return cleanup(cuda_fail(h, e, "cudaMemcpy(graph descriptors)"));
    if ((e = cudaStreamCreateWithFlags(&s0, cudaStreamNonBlocking)) != cudaSuccess)
        return cleanup(cuda_fail(h, e, "cudaStreamCreate"));
    for (size_t i = 0; i < gv.size(); ++i) {
        cudaStream_t s_;
        cudaEvent_t e_;
        if (i + 1 < gv.size()) {
            if ((e = cudaStreamCreateWithFlags(&s_, cudaStreamNonBlocking)) != cudaSuccess)
                return cleanup(cuda_fail(h, e, "cudaStreamCreate"));
            side.push_back(s_);
        }
        if ((e = cudaEventCreateWithFlags(&e_, cudaEventDisableTiming)) != cudaSuccess)
            return cleanup(cuda_fail(h, e, "cudaEventCreate"));
        ev.push_back(e_);
    }
    if ((rc = group_tables(h, gv, s0, &tabv))) return cleanup(rc);
    if ((rc = group_attributes(h, gv, method, vc))) return cleanup(rc);
    if ((e = cudaStreamSynchronize(s0)) != cudaSuccess) return cleanup(cuda_fail(h, e, "table build"));
    if ((e = cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
        return cleanup(cuda_fail(h, e, "cudaStreamBeginCapture"));
    rc = enqueue_groups(h, gv, method, vc, false, g->d_desc, tabv, h->d_grid_sync, s0, side, ev);
    e = cudaStreamEndCapture(s0, &g->graph);
    if (rc) return cleanup(rc);
    if (e != cudaSuccess) return cleanup(cuda_fail(h, e, "cudaStreamEndCapture"));
    if ((e = cudaGraphInstantiate(&g->exec, g->graph, 0)) != cudaSuccess)
        return cleanup(cuda_fail(h, e, "cudaGraphInstantiate"));
    g->kernels = (int)gv.size();
    *out = g;
    return cleanup(OPTIFAX_OK);
}

int optifax_graph_launch(optifax_graph g, void* stream) {
    if (!g || !g->exec) return OPTIFAX_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(g->device) != cudaSuccess) return OPTIFAX_ERR_CUDA;
    return cudaGraphLaunch(g->exec, (cudaStream_t)stream) == cudaSuccess ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

int optifax_graph_kernels(optifax_graph g) { return g ? g->kernels : 0; }

int optifax_opo_run(optifax_handle h, const optifax_opo* cavities, int32_t n_cavities,
                    int32_t variant, int32_t cta_points, optifax_pulse_stats* stats, void* stream) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    if (!cavities || n_cavities < 1) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "no cavities");
    VariantCfg vc;
    if (!variant_cfg(variant, &vc)) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "unknown variant");
    if (cta_points != 0 && (!is_pow2(cta_points) || cta_points < 512 || cta_points > 4096))
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "cta_points must be 0 or a power of two in [512, 4096]");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaSetDevice");
    std::vector<Placed> placed((size_t)n_cavities);
    for (int i = 0; i < n_cavities; ++i) {
        const optifax_opo& cv = cavities[i];
        if (!cv.feedback || !cv.pump) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "feedback and pump are required");
        if (cv.n_trips < 1) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "n_trips must be >= 1");
        if (cv.n_tally < 0 || cv.n_tally > 4 || (cv.n_tally > 0 && !cv.tally_w))
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "n_tally must be 0..4 with tally_w");
        if (cv.steady_trips < 0 || cv.steady_tally < 0 || cv.steady_tally >= 4)
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "bad steady-state settings");
        PulseDev& d = placed[i].d;
        placed[i].want = cta_points;
        int rc = fill_desc(h, cv.pass, vc, &d, stats ? stats + i : nullptr);
        if (rc) return rc;
        d.fb = (const float2*)cv.feedback;
        d.pump = (const float2*)cv.pump;
        d.tally_w = cv.tally_w;
        d.trips = cv.trips;
        d.n_trips = cv.n_trips;
        d.n_tally = cv.n_tally;
        d.steady_trips = cv.steady_trips;
        d.steady_tally = cv.steady_tally;
        d.steady_tol = cv.steady_tol;
        d.hist = (float2*)cv.history;
        if (cv.n_esd < 0 || cv.n_esd > 4 || (cv.n_esd > 0 && (!cv.esd_w || !cv.esd)))
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "n_esd must be 0..4 with esd_w and esd");
        d.esd_w = cv.n_esd > 0 ? cv.esd_w : nullptr;
        d.esd = cv.n_esd > 0 ? cv.esd : nullptr;
        d.n_esd = cv.n_esd;
        d.smt = cv.stepmods_trips;
    }
    std::vector<Group> gv;
    int rc = group_pulses(h, placed, vc.nee ? kHeunNee : OPTIFAX_HEUN, &gv);
    if (rc) return rc;
    return launch_groups(h, gv, OPTIFAX_HEUN, vc, false, (cudaStream_t)stream);
}

int optifax_opo_mex_batch(optifax_handle h,
                          const void* E, const float* alpha_w, const float* G,
                          float w0, double bdiffw0, float step_h, int32_t n_steps, double dt,
                          const float* beta_op, float max_pct_err, float min_pct_err, float sel,
                          const void* Ap_in, const float* stepmods_in,
                          int32_t n_points, int32_t n_pulses, int32_t ap_chunks, int32_t variant,
                          void* A_out, void* Ap_out, float* stepmods_out, void* stream) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    VariantCfg vc;
    if (!variant_cfg(variant, &vc)) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "unknown variant");
    if (n_pulses < 1) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "n_pulses must be >= 1");
    if (!Ap_out || !stepmods_out) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "Ap_out and stepmods_out are required");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaSetDevice");
    cudaStream_t st = (cudaStream_t)stream;
    int method = (variant == OPTIFAX_VARIANT_ODE23) ? OPTIFAX_RK23 : OPTIFAX_HEUN;
    int nchunks = n_chunks_for(n_steps, sel, vc.guard);
    if (nchunks > ap_chunks)
        return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "Ap has fewer chunks than ceil(n_steps/sel)");
    size_t n = (size_t)n_points;
    // outputs start as copies of the inputs (mxGPUCopyFromMxArray, OPO_mex_BATCH.cpp:55-56)
    if (Ap_in && Ap_in != Ap_out) {
        e = cudaMemcpyAsync(Ap_out, Ap_in, sizeof(float2) * n * (size_t)ap_chunks * (size_t)n_pulses,
                            cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return cuda_fail(h, e, "copy Ap");
    }
    if (stepmods_in && stepmods_in != stepmods_out) {
        e = cudaMemcpyAsync(stepmods_out, stepmods_in, sizeof(float) * (size_t)n_steps,
                            cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return cuda_fail(h, e, "copy stepmods");
    }
    std::vector<Placed> placed((size_t)n_pulses);
    for (int b = 0; b < n_pulses; ++b) {
        optifax_pulse p;
        memset(&p, 0, sizeof(p));
        p.n_points = n_points;
        p.n_steps = n_steps;
        p.E_in = (const float2*)E + n * b;
        p.A_out = (float2*)A_out + n * b;
        p.alpha = alpha_w;
        p.beta = beta_op;
        p.G = vc.g_per_pulse ? G + (size_t)n_steps * b : G;
        // reference layout: (b * Nchunks + chunk) * N + i (OPO_CUDA_BATCH_XTAL.cu:302)
        p.Ap = (float2*)Ap_out + (size_t)b * (size_t)nchunks * n;
        p.stepmods = stepmods_out;
        p.w0 = w0; p.h = step_h; p.bdiffw0 = bdiffw0; p.dt = dt;
        p.max_err = max_pct_err; p.min_err = min_pct_err; p.sel = sel;
        placed[b].want = 0;
        int rc = fill_desc(h, p, vc, &placed[b].d, nullptr);
        if (rc) return rc;
    }
    if (n_pulses * (n_points > 4096 ? n_points / 4096 : 1) > 148)
        return fail(h, OPTIFAX_ERR_UNSUPPORTED, "shared-schedule batch larger than one wave of SMs");
    // one size, so one group: every pulse of the shared schedule is in one cooperative grid
    std::vector<Group> gv;
    int rc = group_pulses(h, placed, vc.nee ? kHeunNee : method, &gv);
    if (rc) return rc;
    if (h->cta_points && n_pulses > resident_clusters(h, *find_kernel(gv[0].M, gv[0].C, vc.nee ? kHeunNee : method)))
        return fail(h, OPTIFAX_ERR_UNSUPPORTED, "shared-schedule batch larger than one wave at the handle's cta_points");
    return launch_groups(h, gv, method, vc, n_pulses > 1, st);
}

}  // extern "C"

// chi(3) fibre GNLSE (gnlsefib.m): validation, scratch, descriptors, launch
extern "C" int optifax_gnlse(optifax_handle h, const optifax_gnlse_pulse* pulses, int32_t n_pulses,
                             void* stream) {
    if (!h) return OPTIFAX_ERR_NULL_HANDLE;
    if (!pulses || n_pulses < 1) return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "gnlse: no pulses");
    const int M = pulses[0].n_points, S = pulses[0].n_saves;
    if (M != 512 && M != 1024 && M != 2048 && M != 4096)
        return fail(h, OPTIFAX_ERR_UNSUPPORTED, "gnlse: n_points must be 512, 1024, 2048 or 4096");
    std::vector<GnlseDev> d((size_t)n_pulses);
    for (int i = 0; i < n_pulses; ++i) {
        const optifax_gnlse_pulse& p = pulses[i];
        if (p.n_points != M || p.n_saves != S)
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "gnlse: pulses of one call share n_points and n_saves");
        if (S < 2 || !p.A || !p.B || !p.W || !p.AT_out || !p.AW_out || !(p.length > 0.0) || !(p.dT > 0.0) ||
            !(p.rtol > 0.0) || !(p.atol > 0.0) || !std::isfinite(p.gamma) || !std::isfinite(p.alpha) ||
            !std::isfinite(p.fr) || (p.trace && p.trace_cap < 0))
            return fail(h, OPTIFAX_ERR_INVALID_ARGUMENT, "gnlse: pulse " + std::to_string(i) + " arguments");
        GnlseDev& g = d[(size_t)i];
        memset(&g, 0, sizeof(g));
        g.A = (const float2*)p.A;
        g.B = p.B;
        g.W = p.W;
        g.RW = (p.RW && p.fr != 0.0) ? (const float2*)p.RW : nullptr;
        g.AT_out = (float2*)p.AT_out;
        g.AW_out = (float2*)p.AW_out;
        g.trace = (long long*)p.trace;
        g.trace_cap = p.trace ? p.trace_cap : 0;
        g.max_attempts = p.max_attempts > 0 ? p.max_attempts : 1000000;
        g.stats = p.stats;
        g.gamma = p.gamma; g.fr = p.fr; g.dT = p.dT; g.alpha = p.alpha; g.length = p.length;
        g.rtol = p.rtol; g.atol = p.atol;
        g.n_saves = S;
    }
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t de = cudaSetDevice(h->device);
    if (de != cudaSuccess) return cuda_fail(h, de, "cudaSetDevice");
    int rc = OPTIFAX_OK;
    const Twiddle* quad = get_table(h, h->quadtw, M, M / 4, st, &rc);
    if (!quad) return rc;
    const size_t need_k = (size_t)8 * M * n_pulses;
    if (need_k > h->gnlse_k_cap) {
        size_t cap = h->gnlse_k_cap * sizeof(float2);
        rc = grow_scratch(h, (void**)&h->d_gnlse_k, &cap, need_k * sizeof(float2), st,
                          "cudaMallocAsync(gnlse stage scratch)");
        h->gnlse_k_cap = cap / sizeof(float2);
        if (rc) return rc;
    }
    if ((size_t)n_pulses > h->gnlse_desc_cap) {
        size_t cap = h->gnlse_desc_cap * sizeof(GnlseDev);
        rc = grow_scratch(h, (void**)&h->d_gnlse_desc, &cap, sizeof(GnlseDev) * (size_t)n_pulses, st,
                          "cudaMallocAsync(gnlse descriptors)");
        h->gnlse_desc_cap = cap / sizeof(GnlseDev);
        if (rc) return rc;
    }
    for (int i = 0; i < n_pulses; ++i) d[(size_t)i].K = h->d_gnlse_k + (size_t)8 * M * i;
    rc = order_after_previous(h, st);
    if (rc) return rc;
    cudaError_t e = cudaMemcpyAsync(h->d_gnlse_desc, d.data(), sizeof(GnlseDev) * (size_t)n_pulses,
                                    cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_fail(h, e, "cudaMemcpyAsync(gnlse descriptors)");
    e = launch_gnlse(M, h->d_gnlse_desc, n_pulses, quad, st);
    if (e != cudaSuccess) return cuda_fail(h, e, "gnlse_kernel launch");
    return mark_done(h, st);
}
