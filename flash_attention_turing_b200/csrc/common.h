// Host-side helpers shared by the launchers: error reporting, TMA descriptor creation, the device
// status word.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/fa_b200.h"

namespace fa {

// Records the message returned by fa_last_error() for the calling thread and returns `code`.
int set_error(int code, const std::string& msg);
const std::string& last_error();

#define FA_CHECK_ARG(cond, msg)                                             \
  do {                                                                      \
    if (!(cond)) return ::fa::set_error(FA_ERR_INVALID_ARGUMENT, (msg));    \
  } while (0)

#define FA_CHECK_CUDA(expr)                                                              \
  do {                                                                                   \
    cudaError_t err__ = (expr);                                                          \
    if (err__ != cudaSuccess)                                                            \
      return ::fa::set_error(FA_ERR_CUDA, std::string(#expr) + ": " +                    \
                                              cudaGetErrorString(err__));                \
  } while (0)

// Encodes a rank-4 fp16 tensor map (dims innermost first) with a {64, 1, box_rows, 1} box and the
// 128-byte swizzle.  dims = {d, heads, rows, batch}; strides in elements for heads, rows, batch.
// Returns 0 or a negative FA_ERR_* code (message recorded).
int make_tensor_map_4d(CUtensorMap* map, const void* base, int d, int64_t heads, int64_t rows,
                       int64_t batch, int64_t head_stride, int64_t row_stride, int64_t batch_stride,
                       int box_rows, const char* what);

// Checks that the current device is an sm_100 part; caches the answer per device.
int check_device_sm100();

// Address of the per-device status word kernels write when a bounded wait gives up.
int* device_status_ptr();

// Work counters of the persistent kernels: {next item, finished CTAs} pairs in device memory, all zero between launches (the last CTA of a
// launch to finish puts its pair back to zero).  Two launches that run at the same time must not have the same pair: items would be
// computed by neither.  Launches take the next pair in turn from one of two pools, by whether `stream` is being captured: a captured launch
// keeps its pair for as long as its graph lives, and with a single pool eager launches came round to it.  So two eager launches share a
// pair only with kSchedSlots others issued between them, and two captured ones with kSchedSlots captured between them.
// fa_device_status(1) clears the pools together with a non-zero status word (a launch that gave up on a wait leaves its pair dirty).
constexpr int kSchedSlots = 16384;
int* next_sched_slot(cudaStream_t stream);

// Number of SMs of the current device (cached); 0 on error.
int device_sm_count();

// Launches a kernel that may start before the previous kernel of the stream has finished, as soon as that one lets it
// (grid_launch_dependents() in ptx.cuh): its set-up and launch latency then run under the predecessor.  The kernel has to
// call grid_dependency_wait() before it touches anything the predecessor writes, and in at least one CTA in any case, so
// that its own completion implies that of everything before it.  A kernel that reads, without such a wait, what a kernel further
// back has written (dK/dV: the row statistics) needs its predecessor to wait, fence_acq_rel_gpu() and only then let it start.
template <class Params>
cudaError_t launch_overlapped(void (*kernel)(Params), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                              const Params& params) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, params);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace fa
