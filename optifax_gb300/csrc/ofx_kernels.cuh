// ofx_kernels.cuh -- registry of the compiled (cta_points, cluster, method)
// instantiations of the crystal-pass kernel.  Each ofx_k_*.cu translation
// unit instantiates a subset so the library builds in parallel.
#pragma once
#include <vector>
#include "ofx_pass.cuh"

namespace ofx {

typedef void (*KernelFn)(const PulseDev*, FftTables, KernelCfg);

// rule_only: a shape that the library's own choice of points per CTA may take, not one
// that a caller may ask for.
struct KernelEntry { KernelFn fn; size_t smem; int threads, M, C, method; bool rule_only; };

template <int M, int C, int METH>
KernelEntry kernel_entry(bool rule_only = false) {
    return KernelEntry{&pass_kernel<M, C, METH>, Smem<M, METH, C>::bytes, M / kPoints<M>, M, C, METH, rule_only};
}

void register_kernels_heun_large(std::vector<KernelEntry>& v);
void register_kernels_heun_small(std::vector<KernelEntry>& v);
void register_kernels_rk23(std::vector<KernelEntry>& v);
void register_kernels_heun_nee(std::vector<KernelEntry>& v);

}  // namespace ofx
