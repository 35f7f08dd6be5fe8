// Host calls whose C++ allocations fail, each in turn: a status comes back, no exception
// leaves the library.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

static thread_local int fail_in = 0;  // the n-th allocation of this thread fails
static thread_local bool failed = false;

void* operator new(std::size_t n) {
  if (fail_in > 0 && --fail_in == 0) {
    failed = true;
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main() {
  const size_t n = 600, nao = 300, ngrid = 8000, blk = 64, nblk = ngrid / blk;
  std::vector<double> a(n * n), b(n * n), c(n * n), ao(nao * ngrid), d(nao * nao), rho(ngrid);
  std::vector<uint8_t> tab(nao * nblk);
  for (size_t i = 0; i < tab.size(); i += 3) tab[i] = 1;
  auto gemm = [&] {
    return cfgmm_matmul_anyway_full(c.data(), n * n, a.data(), n * n, b.data(), n * n, n, n, n, n,
                                    n, n, 0, 0);
  };
  auto density = [&] {
    return cfgmm_aodmao2rho_loop_parallel(rho.data(), ngrid, d.data(), nao * nao, ao.data(),
                                          nao * ngrid, ao.data(), nao * ngrid, nao, ngrid, nao,
                                          ngrid, 1, tab.data(), tab.size(), nblk, blk);
  };
  CHECK(gemm() == CFGMM_OK && density() == CFGMM_OK);
  int calls = 0;
  try {
    for (int which = 0; which < 2; ++which)
      for (int nth = 1;; ++nth, ++calls) {
        failed = false;
        fail_in = nth;
        const int rc = which ? density() : gemm();
        fail_in = 0;
        CHECK(rc == CFGMM_OK || rc == CFGMM_ERR_OUT_OF_MEMORY);
        if (!failed) break;  // the call makes fewer allocations
      }
  } catch (const std::bad_alloc&) {
    std::fprintf(stderr, "an exception left the library (call %d)\n", calls);
    return 1;
  }
  return 0;
}
