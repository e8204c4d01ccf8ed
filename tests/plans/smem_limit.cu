// Host-side check of ensure_smem for two threads that ask for different sizes of one kernel at the same time.  The two
// runtime calls it makes are replaced by the ones below: the first thread is held between its limit being set and its caller
// writing that down, for as long as the second thread takes to finish (or a bounded time).  Exit status 0: the limit
// that is in force at the end is the larger of the two.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <cuda_runtime.h>

static std::atomic<int> limit{0}, first_is_set{0}, second_done{0};

static cudaError_t get_device(int* dev) { *dev = 0; return cudaSuccess; }
template <typename K>
static cudaError_t set_attribute(K, cudaFuncAttribute attr, int value) {
  if (attr != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  limit = value;
  if (value == 64 * 1024) {
    first_is_set = 1;
    for (int i = 0; i < 400 && !second_done; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  }
  return cudaSuccess;
}

#define cudaGetDevice get_device
#define cudaFuncSetAttribute set_attribute
#include "../../fgms_b200/csrc/umma.cuh"

__global__ void kernel(int) {}
static std::atomic<int> granted[64];

int main() {
  int rc[2] = {-1, -1};
  std::thread first([&] { rc[0] = fgms::ensure_smem(kernel, 64 * 1024, granted); });
  std::thread second([&] {
    while (!first_is_set) std::this_thread::yield();
    rc[1] = fgms::ensure_smem(kernel, 20 * 1024, granted);
    second_done = 1;
  });
  first.join();
  second.join();
  std::printf("results %d %d, limit in force %d, written down %d\n", rc[0], rc[1], limit.load(), granted[0].load());
  return rc[0] == 0 && rc[1] == 0 && limit == 64 * 1024 && granted[0] == 64 * 1024 ? 0 : 1;
}
