// What belongs to a CUDA context, not to the process: its number, and the
// shared-memory limits of its kernels.
#pragma once

#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <map>
#include <mutex>

#include "qcu_common.cuh"

namespace qcu {

// The driver's number of a context, unique for the life of the process: a device reset gives the device's
// primary context a new one (its handle stays the same, and its memory is gone).  0: no such context.
class ContextId {
 public:
  static unsigned long long current() {
    const Fns& f = fns();
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!f.ok || f.get_current(&c) != CUDA_SUCCESS || !c || f.get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
  }
  static unsigned long long primary(int device) {
    const Fns& f = fns();
    CUdevice d;
    CUcontext c;
    unsigned flags = 0;
    int active = 0;
    unsigned long long id = 0;
    if (!f.ok || f.device(&d, device) != CUDA_SUCCESS || f.state(d, &flags, &active) != CUDA_SUCCESS || !active ||
        f.retain(&c, d) != CUDA_SUCCESS)
      return 0;
    if (f.get_id(c, &id) != CUDA_SUCCESS) id = 0;
    f.release(d);
    return id;
  }

 private:
  struct Fns {
    PFN_cuCtxGetCurrent_v4000 get_current = nullptr;
    PFN_cuCtxGetId_v12000 get_id = nullptr;
    PFN_cuDeviceGet_v2000 device = nullptr;
    PFN_cuDevicePrimaryCtxGetState_v7000 state = nullptr;
    PFN_cuDevicePrimaryCtxRetain_v7000 retain = nullptr;
    PFN_cuDevicePrimaryCtxRelease_v11000 release = nullptr;
    bool ok = true;
    template <typename F>
    void load(F& f, const char* name, unsigned version) {
      void* p = nullptr;
      cudaDriverEntryPointQueryResult q;
      ok &= cudaGetDriverEntryPointByVersion(name, &p, version, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess;
      f = reinterpret_cast<F>(p);
    }
    Fns() {
      load(get_current, "cuCtxGetCurrent", 4000);
      load(get_id, "cuCtxGetId", 12000);
      load(device, "cuDeviceGet", 2000);
      load(state, "cuDevicePrimaryCtxGetState", 7000);
      load(retain, "cuDevicePrimaryCtxRetain", 7000);
      load(release, "cuDevicePrimaryCtxRelease", 11000);
    }
  };
  static const Fns& fns() {
    static const Fns f;
    return f;
  }
};

// Raises a kernel's dynamic shared memory limit before a launch above the
// default 48 KB.  The limit belongs to the kernel in one context: a second
// device of the process, or another context, has its own.
class DynamicSmem {
 public:
  void ensure(const void* kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return;
    const unsigned long long id = ContextId::current();
    std::lock_guard<std::mutex> lk(m_);
    size_t& set = set_[id];
    if (id && bytes <= set) return;
    QCU_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    set = bytes;
  }

 private:
  std::mutex m_;
  std::map<unsigned long long, size_t> set_;  // by context
};

}  // namespace qcu
