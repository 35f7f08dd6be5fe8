// Which split-precision form calls and plans take, on either side of each line.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "../../cfgable-matmul_b200/csrc/aodmao2rho_split.cuh"
#include "../../include/cfgmm.h"
#include "fake_cuda.h"

using cfgmm::split_pair_form;

// the form of a plan of batches of `ngrid` points and the vectors nset each
bool pair_plan(size_t nao, size_t ngrid, std::vector<size_t> nset, size_t nset_max) {
  const size_t blk = 64, nblk = (ngrid + blk - 1) / blk;
  std::vector<double> rho(nset_max * ngrid), ao(nao * ngrid), dms(nset_max * nao * nao);
  std::vector<uint8_t> tab(nao * nblk, 1);
  std::vector<cfgmm_aodm_batch> b;
  for (size_t s : nset) b.push_back({rho.data(), ao.data(), ao.data(), tab.data(), ngrid, ngrid, nblk, s});
  cfgmm_aodm_plan* plan = nullptr;
  CHECK(cfgmm_aodm_plan_create(&plan, b.data(), b.size(), dms.data(), nao, nao, nset_max, blk,
                               CFGMM_PREC_OZAKI_INT8, CFGMM_PLAN_NO_TUNE, nullptr) == CFGMM_OK);
  const bool pair = std::strstr(cfgmm_aodm_plan_info(plan), "\"form\":\"pair\"");
  CHECK(cfgmm_aodm_plan_destroy(plan) == CFGMM_OK);
  return pair;
}

int main() {
  unsetenv("CFGMM_SPLIT_FORM");
  CHECK(split_pair_form(1024, 8192, 1) && !split_pair_form(1024, 8191, 1));
  CHECK(!split_pair_form(1023, 40000, 1) && !split_pair_form(200, 900000, 4));
  CHECK(split_pair_form(2000, 2917, 3) && !split_pair_form(2000, 2916, 3));  // 3.5e10
  setenv("CFGMM_SPLIT_FORM", "pair", 1);
  CHECK(split_pair_form(10, 10, 1) && pair_plan(50, 128, {1}, 1));
  setenv("CFGMM_SPLIT_FORM", "row", 1);
  CHECK(!split_pair_form(4000, 40000, 1) && !pair_plan(1024, 8192, {1}, 1));
  unsetenv("CFGMM_SPLIT_FORM");
  CHECK(pair_plan(1024, 8192, {1}, 1) && !pair_plan(1024, 8128, {1}, 1));
  CHECK(pair_plan(1000, 11667, {3}, 3) && !pair_plan(1000, 11666, {3}, 3));
  // by the batches' own matrices, not by the most that the plan could take
  CHECK(!pair_plan(1000, 11667, {2}, 3));
  CHECK(pair_plan(1000, 1667, std::vector<size_t>(7, 3), 3));   // 5.001e9 per batch
  CHECK(!pair_plan(1000, 1666, std::vector<size_t>(8, 3), 3));  // 4.998e9
  return 0;
}
