// tws_limits.h -- what a launcher remembers of its kernels between launches.
//
// A kernel's dynamic shared memory limit (beyond 48 KB) and its occupancy belong
// to the device that was current when they were set or asked, so they are kept
// per device and kernel: a process that steps grids on a second device sets them
// there too.  No CUDA in here, so that the host tests can compile it alone.
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace tws {

class KernelLimits {
 public:
  // The CTAs of kernel `fn` that an SM of `device` holds with `smem` bytes of dynamic
  // shared memory.  `ask(&ctas)` raises the kernel's limit to `smem` and finds that
  // number; it is called (with the device current) unless it has succeeded before
  // for this kernel on this device with as much.  A failure is returned and not
  // remembered.
  template <class Ask>
  auto get(int device, const void* fn, size_t smem, int* ctas, Ask&& ask) -> decltype(ask(ctas)) {
    using Error = decltype(ask(ctas));
    std::lock_guard<std::mutex> lk(mu_);
    Known& k = known_[{device, fn}];
    if (k.ctas == 0 || k.smem < smem) {
      int n = 0;
      const Error e = ask(&n);
      if (e != Error{}) return e;
      k.smem = smem;
      k.ctas = n > 0 ? n : 1;
    }
    *ctas = k.ctas;
    return Error{};
  }

 private:
  struct Known {
    size_t smem = 0;
    int ctas = 0;
  };
  std::mutex mu_;
  std::map<std::pair<int, const void*>, Known> known_;
};

}  // namespace tws
