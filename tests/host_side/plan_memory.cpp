// A plan's memory comes from cudaMallocAsync, which cudaFree gives back without waiting
// for the work that uses it.  Creates split-precision plans of one batch with each of
// their allocations failing in turn, and destroys plans with a run in flight.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t nao = 1100, ngrid = 8320, blk = 64, nblk = ngrid / blk;
  std::vector<double> rho(ngrid), ao(nao * ngrid), dms(nao * nao);
  std::vector<uint8_t> tab(nao * nblk, 1);
  const cfgmm_aodm_batch one{rho.data(), ao.data(), ao.data(), tab.data(), ngrid, ngrid, nblk, 1};
  cudaStream_t s;
  cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  int row_forms = 0;
  for (int precision : {CFGMM_PREC_FP64, CFGMM_PREC_OZAKI_INT8})
    for (int flags : {CFGMM_PLAN_NO_TUNE, CFGMM_PLAN_NO_TUNE | CFGMM_PLAN_NO_GRAPH})
      for (int nth = 0; nth <= 4; ++nth) {
        cfgmm_aodm_plan* plan = nullptr;
        fake::fail_async_alloc = nth;
        const int rc = cfgmm_aodm_plan_create(&plan, &one, 1, dms.data(), nao, nao, 1, blk,
                                              precision, flags, s);
        fake::fail_async_alloc = 0;
        cudaGetLastError();
        CHECK(fake::free_races == 0);  // cleanup and the fall back to the row form
        CHECK(rc == CFGMM_OK || (rc == CFGMM_ERR_OUT_OF_MEMORY && nth > 0 && !plan));
        if (rc != CFGMM_OK) continue;
        if (precision == CFGMM_PREC_OZAKI_INT8)
          row_forms += !std::strstr(cfgmm_aodm_plan_info(plan), "\"form\":\"pair\"");
        CHECK(cfgmm_aodm_plan_run(plan, s) == CFGMM_OK);
        CHECK(cfgmm_aodm_plan_destroy(plan) == CFGMM_OK);
        CHECK(fake::free_races == 0);
      }
  CHECK(row_forms == 4);  // the pair form's first or second allocation failed, graph or not
  return 0;
}
