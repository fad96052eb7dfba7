// ofx_tmap.cuh -- host side of the tensor-core kernels (ofx_gemm.cu, ofx_fno.cu): tensor
// maps of BF16 operands and the device's error word.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/optifax.h"

namespace ofx_tc {

inline PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    return encode;
}

// rows x cols BF16 row-major with leading dimension ld (elements); box box_rows x 64
inline int make_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, long long ld, int box_rows) {
    auto enc = encoder();
    if (!enc) return OPTIFAX_ERR_CUDA;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? OPTIFAX_OK : OPTIFAX_ERR_CUDA;
}

// Launch with programmatic stream serialisation: the kernel's start overlaps the end of
// the stream's previous kernel (every kernel launched so calls dep_wait before it touches
// global memory).  The surrogate's forward pass is a chain of 14 kernels of 5 us: 100 us for
// one sample by plain launches, 64 so (with the wider lift and projection).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid;
    lc.blockDim = block;
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k, KArgs(args)...);
}

// Device address of the current device's error word (optifax_tc_error), or null
int* error_word();

}  // namespace ofx_tc
