// Host-side plumbing shared by the C-ABI entry points: thread-local error text,
// per-device state (status word), and TMA descriptor encoding through the driver
// entry point (fetched at run time, so the library has no link-time dependency on
// libcuda and loads on a machine without a GPU driver).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/heddle_b200.h"

namespace hb {

int set_error(int code, const char* fmt, ...);
void clear_error();

// Human-readable form of a device status word (0x100 | role: a bounded wait of that role ran out;
// 0x200: shared memory base misaligned).  Returns a pointer to a thread-local buffer.
const char* describe_status(uint32_t word);

#define HB_CUDA_CHECK(expr)                                                                   \
  do {                                                                                        \
    cudaError_t err__ = (expr);                                                               \
    if (err__ != cudaSuccess)                                                                 \
      return hb::set_error(HB_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(err__));   \
  } while (0)

struct DeviceState {
  int device = -1;
  int sm_count = 0;
  int smem_optin = 0;
  int cc = 0;
  uint32_t* status_word = nullptr;  // device memory, zero-initialised
};

// Lazily created state of the CURRENT device (mutex-guarded).  Returns an hb_status.
int get_device_state(DeviceState** out);

// Device facts for entry points that must not allocate: attribute queries and the
// driver entry point only (no cudaMalloc, no per-device state is created).
struct DeviceInfo {
  int device = -1;
  int sm_count = 0;
  int smem_optin = 0;
  int cc = 0;
};
int get_device_info_noalloc(DeviceInfo* out);

// Launches `kernel` so that its start-up (launch latency, barrier and TMEM set-up, descriptor fetch) may run under the tail
// of the stream's previous kernel: programmatic dependent launch.  The kernel calls grid_wait() before it touches memory.
// `cluster` > 0 sets a run-time cluster size.
// Worth it while a kernel's start-up is visible in its time (6 % of a four-kernel train step of 114 us); the attention kernels
// of a long problem start in order instead (`early` false): waiting CTAs cost the step of B4 H32 S4096 0.4 % (2133 -> 2143 us).
inline bool launch_early(double steps_per_cta) { return steps_per_cta <= 100.0; }
template <typename... Params, typename... Args>
inline cudaError_t launch_dependent_if(bool early, void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem,
                                       cudaStream_t stream, unsigned cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2] = {};
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
  if (cluster > 0) {
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = cluster;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                                    unsigned cluster, Args... args) {
  return launch_dependent_if(true, kernel, grid, threads, smem, stream, cluster, args...);
}

// 2-D .. 5-D tiled tensor map with 128-byte swizzle, zero fill out of bounds.
//   dims[i]     extent of dimension i in elements (dimension 0 is contiguous)
//   strides[i]  byte stride of dimension i+1
//   box[i]      tile extent of dimension i in elements
int encode_tensor_map(CUtensorMap* out, CUtensorMapDataType dt, int rank, const void* base, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle,
                      CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_L2_128B);

inline size_t dtype_size(int dtype) { return dtype == HB_FP8_E4M3 ? 1 : 2; }

}  // namespace hb
