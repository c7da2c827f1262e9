// common.h — host-side helpers shared by every translation unit of the library.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "../../include/sgemm_b200.h"

namespace sgb {

// Per-thread status of the most recent public call (sgemm() returns void,
// like the reference, so its outcome is kept here).
void set_last_status(int s);

// Device address of the library's status word (bounded waits write
// SGEMM_B200_ERR_TIMEOUT there).  Resolved once per device.
int* device_status_ptr();

// Cached properties of the current device.
struct DeviceInfo {
    int device = -1;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    size_t smem_optin = 0;
    char name[256] = {0};
};
const DeviceInfo& device_info();

// True when the current device can run sm_100a code.
bool device_is_sm100();

inline cudaStream_t as_stream(sgemm_b200_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// Detail of the most recent failure on this thread (read back through
// sgemm_b200_last_error_detail): printf-style message.
void note_error(const char* fmt, ...);

inline int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return SGEMM_B200_OK;
    note_error("%s: %s", cudaGetErrorName(e), cudaGetErrorString(e));
    if (e == cudaErrorMemoryAllocation) return SGEMM_B200_ERR_NO_MEMORY;
    return SGEMM_B200_ERR_CUDA;
}

// Tensor-map encoding through the driver entry point (no link against libcuda).
bool encode_tensor_map_2d(CUtensorMap* map, CUtensorMapDataType dtype, const void* base,
                          uint64_t inner_elems, uint64_t outer_elems, uint64_t row_stride_bytes,
                          uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle);

// 3-D variant: dims {inner, mid, outer}, byte strides of mid and outer.
bool encode_tensor_map_3d(CUtensorMap* map, CUtensorMapDataType dtype, const void* base,
                          uint64_t inner, uint64_t mid, uint64_t outer, uint64_t mid_stride_bytes,
                          uint64_t outer_stride_bytes, uint32_t box_inner, uint32_t box_mid,
                          uint32_t box_outer, CUtensorMapSwizzle swizzle);

// Library-owned stream-ordered memory pools of the current device; the caller's
// default pool is left untouched.
//  - The library pool: split-path workspaces when the caller passes none, launch
//    tables and host staging.  Its release threshold is unlimited, so freed blocks
//    are reused by the next call instead of going back to the driver.
//  - The scratch pool: operands prepared for a kernel (A transposed, rows copied),
//    which cost a call nothing but speed to do without.  It keeps kScratchKept
//    bytes; what it holds beyond that goes back to the driver at the next
//    synchronisation.
cudaMemPool_t library_pool();
cudaMemPool_t scratch_pool();
// Give back memory of either pool that no stream uses any more.  (cudaFree does, too,
// but the pool goes on counting the memory as used.)
inline void pool_free(void* p) {
    if (!p || cudaFreeAsync(p, (cudaStream_t)0) == cudaSuccess) return;
    cudaGetLastError();
    cudaFree(p);
}

// Most that a call takes to transpose A (16384 x 16384; larger ones are read in
// place), and most that the pool keeps, for such calls on four streams, and all
// plans together hold.  Memory beyond what is kept would be mapped anew by each call
// that is waited for: 20000 x 512 x 20000 takes 7.1 ms, and 45 ms so.
constexpr size_t kScratchPerCall = size_t(1) << 30;
constexpr size_t kScratchKept = size_t(4) << 30;

// Shape checks common to every entry point.  Returns SGEMM_B200_OK or
// SGEMM_B200_ERR_INVALID_ARG.
int check_gemm_args(int m, int n, int k, const float* alpha, const void* A, int lda,
                    const void* B, int ldb, const float* beta, const void* C, int ldc);

inline int div_up(int a, int b) { return (a + b - 1) / b; }

// Launch a kernel that begins with grid_wait() (ptx.cuh), so that its CTAs may
// be placed as soon as those of its predecessor in the stream have ended:
// back to back, a kernel then costs its own time plus about 1 us, where an
// ordinary launch costs about 2.2 us and is rounded up to the next multiple of
// 2.05 us (measured on a B200 with kernels of 1 to 14 us).  Reads and writes
// stay ordered: nothing in global memory is touched before grid_wait()
// returns.  No kernel lets its successor start earlier than that
// (griddepcontrol.launch_dependents): CTAs placed while a grid of about one
// CTA per SM still runs crowd the SMs that are idle or empty first (768^3 on
// 64 x 64 tiles: 35 us per GEMM instead of 24.7 with the release at the
// epilogue, 24 x 4096 x 4096 on 32 x 32 tiles 62 instead of 42 with it at the
// start).
// `cluster`: CTAs per thread-block cluster.
template <class... P, class... A>
inline cudaError_t launch_chained_cluster(int cluster, void (*kernel)(P...), int grid, int threads,
                                          size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), int grid, int threads, size_t smem,
                                  cudaStream_t stream, A... args) {
    return launch_chained_cluster(1, kernel, grid, threads, smem, stream, args...);
}

}  // namespace sgb
