// Host calls on two devices from two threads: while the first device's kernels run, the
// second device's call goes through.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <future>
#include <thread>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int product(int dev, size_t n) {  // pageable arrays large enough for the pinned buffers
  cudaSetDevice(dev);
  std::vector<double> a(n * n), b(n * n), c(n * n);
  return cfgmm_matmul_anyway_full(c.data(), n * n, a.data(), n * n, b.data(), n * n, n, n, n, n, n,
                                  n, 0, 0);
}

int main() {
  CHECK(product(0, 500) == CFGMM_OK && product(1, 500) == CFGMM_OK);
  fake::long_device = 0;
  std::thread first([] { CHECK(product(0, 600) == CFGMM_OK); });
  while (!fake::running()) std::this_thread::yield();
  std::this_thread::sleep_for(std::chrono::milliseconds(200));  // it waits for its kernels
  auto second = std::async(std::launch::async, [] { return product(1, 600); });
  CHECK(second.wait_for(std::chrono::seconds(20)) == std::future_status::ready);
  CHECK(second.get() == CFGMM_OK);
  fake::release();
  first.join();
  return 0;
}
