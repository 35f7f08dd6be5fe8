// A call that ran out of device memory says so, and the next one is not told of it again.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t n = 200, nblk = 4, blk = 50;
  std::vector<float> a(n * n), b(n * n), c(n * n);
  std::vector<double> d(n * n), rho(n), ao(n * n);
  std::vector<uint8_t> tab(n * nblk, 1);
  auto product = [&] {
    return cfgmm_matmul_f32_dev(c.data(), a.data(), b.data(), n, n, n, n, n, n, 0, 0,
                                CFGMM_PREC_FP64, nullptr);
  };
  const cfgmm_aodm_batch one{rho.data(), ao.data(), ao.data(), tab.data(), n, n, nblk, 1};
  auto plan = [&] {
    cfgmm_aodm_plan* p = nullptr;
    const int rc = cfgmm_aodm_plan_create(&p, &one, 1, d.data(), n, n, 1, blk, CFGMM_PREC_FP64,
                                          CFGMM_PLAN_NO_TUNE, nullptr);
    cfgmm_aodm_plan_destroy(p);
    return rc;
  };
  for (int turn = 0; turn < 2; ++turn) {
    fake::fail_async_alloc = 1;
    CHECK((turn ? plan() : product()) == CFGMM_ERR_OUT_OF_MEMORY);
    CHECK((turn ? product() : plan()) == CFGMM_OK);
  }
  return 0;
}
