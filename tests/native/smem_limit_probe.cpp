// allow_smem (csrc/ftk_host.cuh) from two threads at once, with a stand-in for the CUDA runtime:
// cudaFuncSetAttribute sets a limit that may go down as well as up.  The thread that asks for the
// smaller size is held inside its call until the other one's has returned, or for 200 ms where
// that one waits for it.  Prints what the limit and a later look at the record come to.
#include <cuda_runtime.h>

// as nvcc has it: a kernel instead of a pointer to void
template <typename... Params>
cudaError_t cudaFuncSetAttribute(void (*kernel)(Params...), cudaFuncAttribute attribute, int value) {
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), attribute, value);
}

#include "ftk_host.cuh"

#include <chrono>
#include <cstdio>
#include <thread>

static std::atomic<int> limit{0}, calls{0};
static std::atomic<bool> small_inside{false}, large_done{false};
constexpr size_t SMALL = 99328, LARGE = 214016;

extern "C" cudaError_t cudaGetDevice(int* dev) {
  *dev = 0;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int value) {
  calls++;
  if (value == static_cast<int>(SMALL)) {
    small_inside = true;
    for (int i = 0; i < 200 && !large_done; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  }
  limit = value;
  return cudaSuccess;
}

static void kernel(int) {}

int main() {
  int bad = 0;
  std::thread a([&] { bad |= ftk::allow_smem<kernel>(SMALL); });
  while (!small_inside) std::this_thread::yield();
  std::thread b([&] {
    bad |= ftk::allow_smem<kernel>(LARGE);
    large_done = true;
  });
  a.join();
  b.join();
  // every size that was allowed fits, without another call
  const int before = calls;
  bad |= ftk::allow_smem<kernel>(SMALL) | ftk::allow_smem<kernel>(LARGE);
  std::printf("%d %d %d\n", bad, limit.load(), calls - before);
}
