// Shared between the translation units of libpk100: status codes, enums that are
// also part of the C ABI (see include/pk100.h) and the launch-status helper.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "../../include/pk100.h"

// Maps the sticky-free launch error of the last kernel launch to the ABI's
// convention: 0 ok, positive = CUDA runtime error code.
// Number of kernels launched through this library by the calling process (monotonic).
extern "C" long long pk100_launch_count(void);
void pk100_count_launch();

static inline int pk100_launch_status() {
    const cudaError_t err = cudaPeekAtLastError();
    if (err == cudaSuccess) {
        pk100_count_launch();
        return PK100_OK;
    }
    cudaGetLastError();   // clear the non-sticky launch error so later calls are not poisoned
    return static_cast<int>(err);
}

// What belongs to one device is remembered per device (a process may drive several, from several threads); devices
// behind the table are asked each time.
constexpr int kPk100Devices = 64;

// Lets `Kernel` use `bytes` of dynamic shared memory on the current device.
template <auto Kernel>
static inline cudaError_t pk100_grant_smem(int bytes) {
    static std::atomic<bool> granted[kPk100Devices];
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < kPk100Devices && granted[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    err = cudaFuncSetAttribute(reinterpret_cast<const void*>(Kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (err == cudaSuccess && dev < kPk100Devices) granted[dev].store(true, std::memory_order_relaxed);
    return err;
}

// SMs of the current device (148 where it cannot be asked).
inline int pk100_sm_count() {
    static std::atomic<int> counts[kPk100Devices];
    int dev = 0, count = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev < kPk100Devices && (count = counts[dev].load(std::memory_order_relaxed)) > 0) return count;
    if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || count <= 0) return 148;
    if (dev < kPk100Devices) counts[dev].store(count, std::memory_order_relaxed);
    return count;
}

// Programmatic dependent launch for the kernels of the per-block chain (LayerNorm, GEMMs,
// attention, depthwise convolution).  Each of them issues griddepcontrol.launch_dependents on
// entry and griddepcontrol.wait before its first access to global memory, so a launch made with
// the attribute below may become resident while its predecessor in the stream drains: the launch
// latency and the prologue (barrier set-up, tensor-memory allocation, descriptor prefetch) leave
// the critical path; the data dependency is still the whole predecessor grid.  On by default;
// pk100_set_dependent_launch(0) restores plain stream order.
//
// A chain of such launches reaches further back than its last link: every kernel lets the next one start
// before it has itself waited, so the prologue of the n-th may run while whatever stands in front of the
// first still does.  What a prologue reads (weights, geometry: b_settled, constants_settled below) must
// therefore have been written in front of a PLAIN launch that opens the chain; pk100_run_layers and the
// subsampling stage open theirs with one.
bool pk100_dependent_launch_enabled();

// dependent: as above where enabled; false = plain stream order for this launch
template <typename... Params, typename... Args>
static inline void pk100_launch(bool dependent, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem_bytes,
                                cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = dependent && pk100_dependent_launch_enabled() ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
static inline void pk100_launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem_bytes,
                                        cudaStream_t stream, Args&&... args) {
    pk100_launch(true, kernel, grid, block, smem_bytes, stream, args...);
}

// Row geometry of a batch: uniform blocks of seg_stride rows per utterance (tiles == nullptr), or a packed
// batch in which every utterance takes whole 128-row tiles: tiles[row / 128] = {first row of the tile's
// utterance, its valid rows}.
struct pk100_rows {
    const int2* tiles;
    int seg_stride, valid_rows;
    const int* seg_valid;
};

// The row-wise operators behind the C entry points, on either geometry (total_rows: a multiple of 128 when
// packed).  Arguments are the entry points', already checked (pointers of the depthwise form excepted: it
// checks them itself).  dependent = false opens a chain (see above).
int pk100_layer_norm_rows(void* stream, const void* input, const void* gamma, const void* beta, void* output, float* scales,
                          int mode, float inv_scale, int total_rows, const pk100_rows& geometry, float eps, bool dependent = true);
int pk100_layer_norm_pair_rows(void* stream, const void* input, const void* gamma, const void* beta, void* output,
                               const void* next_gamma, const void* next_beta, void* next_output, float* next_scales,
                               int next_mode, float next_inv_scale, int total_rows, const pk100_rows& geometry, float eps);
int pk100_depthwise_bn_silu_rows(void* stream, const void* input, const void* dw_weight, const float* bn_gamma, const float* bn_beta,
                                 const float* bn_mean, const float* bn_var, void* output, float* row_scales, int quantize,
                                 int total_rows, int segments, const pk100_rows& geometry, float eps);

// Local attention behind pk100_local_relpos_attention_tcgen05 on either geometry (total_rows: a multiple of 128).
// constants_settled: position, biases and geometry were written in front of the plain launch that opened the chain.
int pk100_local_attention_rows(void* stream, const void* query, int ldq, const void* key, int ldk, const void* value, int ldv,
                               const void* position, const void* bias_u, const void* bias_v, void* output, int ldo,
                               int total_rows, const pk100_rows& geometry, bool constants_settled, int* status);

// pk100_gemm; b_settled: B was written in front of the plain launch that opened the chain.
int pk100_gemm_chained(void* stream, const pk100_gemm_args* args, bool b_settled);

// SMs a launch may count on: all of them, or the cap set by pk100_set_gemm_cta_cap.
int pk100_cta_budget();

// 2-D TMA descriptor of a row-major matrix [rows, cols] (`ld` elements between rows) with a box of
// [box_rows, swizzle_bytes / elem_bytes] elements; served from the library's descriptor cache
// (gemm_host.cu).  `map` points to a CUtensorMap.
int pk100_tensor_map_2d(void* map, const void* base, int elem_bytes, unsigned long long rows,
                        unsigned long long cols, unsigned long long ld, int box_rows, int swizzle_bytes);
