// Host-side helper: one-time set-up per DEVICE.
//
// cudaFuncSetAttribute (opt-in to more than 48 KiB of dynamic shared memory) belongs to the current device's
// context, so a process that calls the library on cuda:0 and later on cuda:1 has to set it on each.  A
// DeviceOnce keeps one flag per device ordinal under a mutex; `run` calls the set-up function the first time it
// sees the current device and afterwards returns that device's cached result.  The first use on a device also
// checks that it is an sm_100 part (compute capability 10.x): the kernels are built for sm_100a only.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "kda_b200.h"

namespace kda {

constexpr int kMaxDeviceOrdinals = 64;

struct DeviceOnce {
  std::mutex mu;
  bool done[kMaxDeviceOrdinals] = {};
  int result[kMaxDeviceOrdinals] = {};

  // Returns KDA_OK, KDA_E_DEVICE (not an sm_100 device), KDA_E_LIMIT (device ordinal beyond the table) or a
  // positive cudaError_t.  `setup` returns a cudaError_t and runs with the device current.
  template <class F>
  int run(F&& setup) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 0 || dev >= kMaxDeviceOrdinals) return KDA_E_LIMIT;
    std::lock_guard<std::mutex> lk(mu);
    if (!done[dev]) {
      int major = 0;
      e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
      if (e != cudaSuccess) return static_cast<int>(e);
      if (major != 10) {
        result[dev] = KDA_E_DEVICE;
      } else {
        e = setup();
        result[dev] = static_cast<int>(e);
      }
      done[dev] = true;
    }
    return result[dev];
  }
};

// Launches a kernel of a call behind the previous kernel of the same call: its CTAs may be brought up while that one's last CTAs still
// run (programmatic dependent launch), which hides the launch latency and the drain.  Such a kernel starts with chain_point(), before
// it touches memory or asks for tensor memory: that is where it waits for everything in front of it.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// SMs of the current device (asked once per device)
inline int sm_count() {
  static std::atomic<int> known[kMaxDeviceOrdinals];
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess) return sms;
  const bool keep = dev >= 0 && dev < kMaxDeviceOrdinals;
  if (keep && known[dev].load(std::memory_order_relaxed) > 0) return known[dev].load(std::memory_order_relaxed);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (keep) known[dev].store(sms, std::memory_order_relaxed);
  return sms;
}

}  // namespace kda
