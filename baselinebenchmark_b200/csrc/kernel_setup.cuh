// What the host asks the runtime about a device and a kernel, or tells it about a kernel, once instead of at every launch.
// None of it depends on a call's inputs.  The sizes of a device are kept per device.  What is set on a kernel is kept per context: it
// belongs to the module that is loaded there, and a caller may make another context of the device current or reset the device.
// Contexts are told apart by the number that the driver gives each of them and never gives again (a device that was reset has
// a new one at the old address).  Fixed tables: nothing here allocates; what does not fit is asked for every time.
// With the settings made at every launch a decode step behind 20011 tokens, 16/4 heads, head dim 64, which waits for the host, took 37.4 us in
// place of 36.7 (means of three runs in turn, which differ by 0.4).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

namespace moba {

struct DeviceInfo {
  int sms, smem_per_sm, regs_per_sm;
};

class KernelSetup {
 public:
  // Defined in one source file and not here: the static object of an inline function is one for the whole process, also for two builds
  // of this library that are loaded side by side and may not agree on what it looks like.
  static KernelSetup& instance();
  // Of the current device.
  DeviceInfo device() {
    DeviceInfo info{148, 0, 0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return info;
    std::lock_guard<std::mutex> lock(mutex_);
    const bool kept = dev >= 0 && dev < kDevices;
    if (kept && devices_[dev].known) return devices_[dev].info;
    const bool ok = cudaDeviceGetAttribute(&info.sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
                    cudaDeviceGetAttribute(&info.smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess &&
                    cudaDeviceGetAttribute(&info.regs_per_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev) == cudaSuccess;
    if (kept && ok) devices_[dev] = Device{true, info};
    return info;
  }
  // Allows `kernel` that much dynamic shared memory in the current context.  `regs`: its registers per thread; `carveout`: the SM's
  // memory is to be shared memory, all of it.
  cudaError_t prepare(const void* kernel, size_t smem, int* regs, bool carveout) {
    std::lock_guard<std::mutex> lock(mutex_);
    Kernel unkept{};
    Kernel* k = place(context_number(), kernel);
    if (k == nullptr) k = &unkept;
    cudaError_t e;
    if (smem > k->smem) {
      if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
      k->smem = smem;
    }
    if (carveout && !k->carveout) {
      if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100)) != cudaSuccess) return e;
      k->carveout = true;
    }
    if (regs != nullptr) {
      if (k->regs == 0) {
        cudaFuncAttributes attr;
        if ((e = cudaFuncGetAttributes(&attr, kernel)) != cudaSuccess) return e;
        k->regs = attr.numRegs;
      }
      *regs = k->regs;
    }
    return cudaSuccess;
  }

 private:
  static constexpr int kDevices = 64, kContexts = 16, kKernels = 256;   // (some 100 kernels of the library ask)
  struct Device {
    bool known;
    DeviceInfo info;
  };
  struct Kernel {
    const void* kernel;
    size_t smem;
    int regs;
    bool carveout;
  };
  struct Context {
    unsigned long long number;
    Kernel kernels[kKernels];
  };
  typedef CUresult (*GetCurrentFn)(CUcontext*);
  typedef CUresult (*GetNumberFn)(CUcontext, unsigned long long*);

  KernelSetup() {
    void *current = nullptr, *number = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &current, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess ||
        cudaGetDriverEntryPoint("cuCtxGetId", &number, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      return;
    get_current_ = reinterpret_cast<GetCurrentFn>(current);
    get_number_ = reinterpret_cast<GetNumberFn>(number);
  }
  // Of the current context; 0 where there is none yet, or none any more.
  unsigned long long context_number() const {
    CUcontext c = nullptr;
    unsigned long long number = 0;
    if (get_number_ == nullptr || get_current_(&c) != CUDA_SUCCESS || c == nullptr || get_number_(c, &number) != CUDA_SUCCESS) return 0;
    return number;
  }
  // The kernel's place in the context's table, null when there is none.  A context that is new here takes the table
  // of the one that came first.
  Kernel* place(unsigned long long number, const void* kernel) {
    if (number == 0) return nullptr;
    int c = 0;
    while (c < kContexts && contexts_[c].number != number) ++c;
    if (c == kContexts) {
      c = next_;
      next_ = (next_ + 1) % kContexts;
      contexts_[c] = Context{};
      contexts_[c].number = number;
    }
    const size_t at = (((uintptr_t)kernel >> 4) * 0x9E3779B9u) >> 8;
    for (int i = 0; i < kKernels; ++i) {
      Kernel& k = contexts_[c].kernels[(at + i) % kKernels];
      if (k.kernel == kernel) return &k;
      if (k.kernel == nullptr) {
        k.kernel = kernel;
        return &k;
      }
    }
    return nullptr;
  }
  std::mutex mutex_;
  GetCurrentFn get_current_ = nullptr;
  GetNumberFn get_number_ = nullptr;
  int next_ = 0;
  Device devices_[kDevices] = {};
  Context contexts_[kContexts] = {};
};

inline DeviceInfo device_info() { return KernelSetup::instance().device(); }
template <typename K>
inline cudaError_t prepare_kernel(K* kernel, size_t smem, int* regs = nullptr, bool carveout = false) {
  return KernelSetup::instance().prepare(reinterpret_cast<const void*>(kernel), smem, regs, carveout);
}

}  // namespace moba
