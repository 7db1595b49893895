// Two threads make the library's first use of the tensor-map encoder at once.
// The driver's entry point is replaced by one that takes a while to be found,
// so no device is needed; both threads have to get it.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

static std::atomic<int> lookups{0};
static cudaError_t slow_lookup(const char *, void **p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *q) {
  ++lookups;
  std::this_thread::sleep_for(std::chrono::milliseconds(200));
  *p = reinterpret_cast<void *>(1);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
#define cudaGetDriverEntryPointByVersion slow_lookup
#include "cgx.cu"

int main() {
  bool found[2] = {false, false};
  std::thread first([&] { found[0] = tma_encoder() != nullptr; });
  while (!lookups) std::this_thread::yield();
  found[1] = tma_encoder() != nullptr;
  first.join();
  printf("%d %d\n", found[0], found[1]);
  return found[0] && found[1] ? 0 : 1;
}
