// Library-wide pieces of the C interface: the per-thread error message and a version probe.

#include <stdarg.h>
#include <stdio.h>

#include <mutex>
#include <unordered_set>

#include "tensor_map.cuh"

static thread_local char g_last_error[512] = "";

int gk_fail(int status, const char* fmt, ...) {
    va_list args;
    va_start(args, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, args);
    va_end(args);
    return status;
}

int g_gk_pdl = -1;

// Every kernel asks for the largest shared-memory share of the SM's L1/shared-memory array.  An SM changes
// that split only when it is idle, so kernels that prefer different splits cannot be resident side by side,
// and a kernel launched early (programmatic dependent launch) would wait for the SMs to drain instead of
// fetching its weights next to the kernel in front of it.
void gk_prepare_kernel(const void* kernel) {
    static std::mutex lock;
    static std::unordered_set<const void*> seen;
    std::lock_guard<std::mutex> guard(lock);
    if (seen.insert(kernel).second)
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

// Switches programmatic dependent launch on (1) or off (0) for every later kernel launch of the library, or leaves it to those behind the
// first of a layer or of a call (-1); returns the previous setting.
GK_EXPORT int gk_set_pdl(int on) {
    const int before = g_gk_pdl;
    g_gk_pdl = on < 0 ? -1 : on ? 1 : 0;
    return before;
}

thread_local int t_gk_chain = 0;

// 1: the calls of this thread up to the one with 0 launch the kernels of one layer, which read nothing before pdl_wait() that one of
// them writes; all but the first may start early.  -1: up to the next call of this none of the thread's kernels starts early, whatever the
// switch says.  Returns the state before (0: neither, 2: behind the first of a layer), which may be put back.
GK_EXPORT int gk_chain(int state) {
    const int before = t_gk_chain;
    t_gk_chain = state;
    return before;
}

// `bytes` from pinned host memory to the device, in stream order.
GK_EXPORT int gk_copy_to_device(void* dst, const void* src, long long bytes, void* stream) {
    const cudaError_t err = cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream);
    if (err != cudaSuccess) return gk_fail(GK_CUDA_ERROR, "copy_to_device: %s", cudaGetErrorString(err));
    return GK_OK;
}

GK_EXPORT const char* gk_last_error() { return g_last_error; }

// Interface revision: the Python side refuses a library built from other sources.
GK_EXPORT int gk_interface_version() { return 1; }

// Compute capability of the current device as major * 10 + minor, or a negative CUDA error.
GK_EXPORT int gk_device_capability() {
    int device = 0, major = 0, minor = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device);
    if (err != cudaSuccess) return -(int)err;
    return major * 10 + minor;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

int gk_matrix_map(CUtensorMap* map, const void* base, long long rows, int k, long long ld, int box_k, int box_rows, bool swizzle) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return gk_fail(GK_CUDA_ERROR, "the driver does not offer cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(__nv_bfloat16)};
    cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return gk_fail(GK_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return GK_OK;
}
