// Host-side helpers shared by every translation unit of libb200ait:
// thread-local last-error text, exception -> status conversion, the per-device
// status word that kernels write when a bounded wait gives up.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <stdexcept>
#include <string>
#include <utility>

#define B200AIT_EXPORT extern "C" __attribute__((visibility("default")))

namespace b200ait {

void set_last_error(const std::string& msg);
const std::string& last_error();

// device pointer to this device's int status word (allocated on first use, zeroed)
int* device_status_word();

// Process-wide count of kernels this library has launched (every launch site calls count_launch();
// a launch made while a stream is being captured counts once, at capture).
extern std::atomic<uint64_t> g_kernel_launches;
inline void count_launch() { g_kernel_launches.fetch_add(1, std::memory_order_relaxed); }

// number of SMs of the current device (cached per device)
int sm_count();

// Raises a kernel's dynamic shared-memory limit once per device (bit i of `done` = device i).
void opt_in_smem_once(std::atomic<uint64_t>& done, const void* kernel, int bytes);

struct Error : public std::runtime_error {
  using std::runtime_error::runtime_error;
};

#define B200AIT_CUDA_CHECK(expr)                                                              \
  do {                                                                                        \
    cudaError_t _e = (expr);                                                                  \
    if (_e != cudaSuccess) {                                                                  \
      throw ::b200ait::Error(std::string(#expr " failed: ") + cudaGetErrorString(_e));        \
    }                                                                                         \
  } while (0)

#define B200AIT_REQUIRE(cond, msg)                       \
  do {                                                   \
    if (!(cond)) throw ::b200ait::Error(std::string(msg)); \
  } while (0)

// Launches a kernel in clusters of `cluster` CTAs. With `early` its CTAs may become resident while the kernel ahead of it on the
// stream still runs, and wait there (grid_wait in ptx.cuh, which such a kernel has to call) until that one has finished and
// its writes can be seen: the launch and the kernel's own set-up are then over when the data is ready. Between two launches of
// the tile GEMM that is worth 0.5 .. 0.8 us (154 x 320 x 768: 4.6 -> 3.8 us, 384 x 768 x 768 + add: 5.0 -> 4.2). The other kernels
// (one to four rows of X, the sum of split K, unaligned GEMMs, rows that a warp cannot hold in 16-byte pieces, reductions over an
// inner dimension, attention without tensor cores) are launched with <<<>>>: an early launch of them has not been measured.
template <class... Params, class... Args>
void launch_early(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, bool early,
                  unsigned cluster, Args&&... args) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  if (early) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  count_launch();
  B200AIT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

// Is this launch being captured into a graph? (Of a stream that cannot be asked: no.)
inline bool in_capture(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return status == cudaStreamCaptureStatusActive;
}

// Runs `fn`, converts any exception into a nonzero status + last-error text.
template <class F>
int guarded(const char* where, F&& fn) {
  try {
    fn();
    return 0;
  } catch (const std::exception& e) {
    set_last_error(std::string(where) + ": " + e.what());
    return 1;
  } catch (...) {
    set_last_error(std::string(where) + ": unknown error");
    return 1;
  }
}

enum DType : int { kDTypeHalf = 1, kDTypeFloat = 2, kDTypeInt = 3, kDTypeBFloat16 = 6 };  // values of AITemplateDtype

}  // namespace b200ait
