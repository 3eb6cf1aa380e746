// Shared host-side helpers of libaiter_b200.so: error bridging of the C-ABI, tensor checks.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <sstream>
#include <stdexcept>
#include <string>
#include <utility>

#include "../../include/aiter_b200.h"

namespace b200 {

// Thread-local message of the last failed call (same contract as the reference's
// g_aiter_last_error, csrc/include/aiter_ctypes_error.h:61-71). Defined in abi.cu.
std::string& last_error();

template <typename... Args>
[[noreturn]] inline void fail(Args&&... args) {
    std::ostringstream os;
    (os << ... << args);
    throw std::runtime_error(os.str());
}

#define B200_CHECK(cond, ...)                         \
    do {                                              \
        if (!(cond)) ::b200::fail(__VA_ARGS__);       \
    } while (0)

#define B200_CUDA(expr)                                                                   \
    do {                                                                                  \
        cudaError_t e_ = (expr);                                                          \
        if (e_ != cudaSuccess)                                                            \
            ::b200::fail(#expr, " failed: ", cudaGetErrorName(e_), " (", cudaGetErrorString(e_), ")"); \
    } while (0)

// Runs fn, converts any C++ exception into status -1 + thread-local message; exceptions never
// cross the C boundary.
template <typename Fn>
inline int safe_call(Fn&& fn) {
    last_error().clear();
    try {
        fn();
        return 0;
    } catch (const std::exception& e) {
        last_error() = e.what();
        return -1;
    } catch (...) {
        last_error() = "unknown C++ exception";
        return -1;
    }
}

inline bool is_contiguous(const aiter_tensor_t* t) {
    if (t->numel_ == 0) return true;
    int64_t expected = 1;
    for (int d = t->ndim - 1; d >= 0; --d) {
        if (t->shape[d] != 1 && t->strides[d] != expected) return false;
        expected *= t->shape[d];
    }
    return true;
}

inline void check_tensor(const aiter_tensor_t* t, const char* name, int dtype, int ndim) {
    B200_CHECK(t != nullptr, name, " must not be NULL");
    B200_CHECK(t->ndim >= 0 && t->ndim <= 8, name, ": bad ndim ", t->ndim);
    B200_CHECK(t->device_id >= 0, name, " must be a CUDA tensor");
    B200_CHECK(dtype < 0 || t->dtype_ == dtype, name, ": unexpected dtype code ", t->dtype_,
               " (want ", dtype, ")");
    B200_CHECK(ndim < 0 || t->ndim == ndim, name, ": expected ", ndim, " dims, got ", t->ndim);
    B200_CHECK(is_contiguous(t), name, " must be contiguous");
    B200_CHECK(t->numel_ == 0 || t->ptr != nullptr, name, ": NULL data pointer");
}

// Programmatic dependent launch: the grid may be placed while its predecessor on the stream still runs; the kernel calls
// pdl_wait() before it touches anything an earlier kernel wrote or reads. Every kernel calls pdl_wait() somewhere, so a
// grid's completion implies the completion of all before it. Most trigger their successor (pdl_trigger) after their own
// wait; then, when the successor starts, everything before the triggering kernel is complete, and only that kernel may still
// run. What works before its own wait relies on this and names the kernel it may run beside: the fill of the two-kernel sort
// (its predecessor is always the count kernel, whose sorting CTAs trigger after their wait) and the layer's activation
// quantiser (its predecessor is always the sort). That quantiser triggers BEFORE its wait, so whatever is launched behind it
// must wait before it touches anything (stage 1 and the per_Tensor kernels do). The launch over the single blocks of a stage, whose
// predecessor is always the launch over its pairs, waits at its end only and triggers before, so the same holds for its successors
// (the requantisers, stage 2's pairs, the final rounding). A stage-2 launch that leaves SMs idle does not
// trigger at all: its successor starts when it is over. Saves the 1-2 us between two dependent short kernels and hides their start-up.
template <typename... Params, typename... Args>
inline void launch_kernel(bool overlap, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                          Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (overlap) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)cluster;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}
template <typename... Params, typename... Args>
inline void launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    launch_kernel(true, kernel, grid, block, smem, stream, 1, std::forward<Args>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// Row blocks of a sorted buffer (128 rows each), split for the GEMM stages: two neighbouring blocks of one expert are a pair,
// the last block of an expert with an odd number of them is single. Written by the sort, all pointers on the device.
struct BlockLists {
    int* counts = nullptr;    // {pairs, singles}
    int* pairs = nullptr;     // first block of each pair
    int* singles = nullptr;
    int64_t max_pairs = 0, max_singles = 0;   // bounds the host knows
};

// One GEMM stage over activation rows in sorted order (moe_gemm_sorted.cu)
struct SortedStage {
    const void* rows;          // [P, K] fp8
    const float* a_scale;      // [ceil(K/512)][ld][4]; rowwise: [P], or [1] with a_scale_ld 0
    const void* w;
    const float* w_scale;
    void* out;                 // stage 1: [P, I] bf16; stage 2: acc [M, H]
    const int* sorted_ids;
    const float* sorted_w;
    const int* sorted_eids;
    const int* num_valid;
    unsigned* amax;
    int* status;
    BlockLists lists;
    int64_t M, H, I, E, P;     // E: experts of the weights
    int ld;                    // row pitch of block scales
    int a_scale_ld, w_scale_by_expert, use_weight, activation, device;
    bool rowwise;
};

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        B200_CUDA(cudaGetDevice(&prev));
        if (prev != dev) B200_CUDA(cudaSetDevice(dev));
        else prev = -1;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

inline int sm_count(int dev) {
    static int cached[64] = {0};
    if (dev < 64 && cached[dev] > 0) return cached[dev];
    int n = 0;
    B200_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    if (dev < 64) cached[dev] = n;
    return n;
}

}  // namespace b200
