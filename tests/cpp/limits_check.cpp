// Launch limits on two devices (csrc/tws_limits.h) against a driver that keeps a
// kernel's shared memory limit per device, as CUDA does.
#include <cstdio>

#include "tws_limits.h"

namespace {

constexpr int kOk = 0, kRefused = 1;
char kernels[2];
size_t limit[2][2] = {{48 << 10, 48 << 10}, {48 << 10, 48 << 10}};  // [device][kernel]
int asked = 0;

// Raises the limit where `works`, and a launch with `smem` bytes.
int launch(tws::KernelLimits& l, int device, int kernel, size_t smem, bool works = true) {
  int ctas = 0;
  const int e = l.get(device, &kernels[kernel], smem, &ctas, [&](int* n) {
    ++asked;
    if (!works) return kRefused;
    limit[device][kernel] = smem;
    *n = (int)((227u << 10) / smem);
    return kOk;
  });
  if (e != kOk) return e;
  if (ctas != (int)((227u << 10) / smem)) return 3;
  return smem <= limit[device][kernel] ? kOk : 2;
}

}  // namespace

#define CHECK(x)                                           \
  do {                                                     \
    if (!(x)) {                                            \
      std::printf("line %d: %s\n", __LINE__, #x);          \
      return 1;                                            \
    }                                                      \
  } while (0)

int main() {
  tws::KernelLimits l;
  CHECK(launch(l, 0, 0, 72 << 10) == kOk && asked == 1);
  CHECK(launch(l, 0, 0, 72 << 10) == kOk && asked == 1);  // once per device
  CHECK(launch(l, 1, 0, 72 << 10) == kOk && asked == 2);  // a second device has its own
  CHECK(launch(l, 1, 1, 60 << 10) == kOk && asked == 3);  // and so has another kernel
  CHECK(launch(l, 1, 1, 90 << 10) == kOk && asked == 4);  // a larger launch raises it
  CHECK(launch(l, 0, 1, 90 << 10, false) == kRefused && asked == 5);
  CHECK(launch(l, 0, 1, 90 << 10) == kOk && asked == 6);  // a failure is not remembered
  return 0;
}
