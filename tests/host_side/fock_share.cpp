// The Fock kernel's sharing of its work: every weight vector in one group, groups of at
// most four, and the items' total exact where it passes 2^31 (2^25 items of one-point
// blocks, 300 vectors).
#include <cstdio>
#include <cstdlib>

#include <cuda_runtime.h>

#include "../../cfgable-matmul_b200/csrc/fock.cuh"
#include "fake_cuda.h"

int main() {
  const int ctas = 296;
  for (int items : {0, 1, 7, 275, 789, 790, 2368, 2369, 100000, 1 << 25, 2147483647})
    for (int nset : {1, 2, 3, 4, 5, 9, 300, 70000}) {
      const cfgmm::FockShare s = cfgmm::fock_share(items, nset, ctas);
      CHECK(s.groups >= 1 && s.groups <= nset && s.per_group >= 1 && s.per_group <= 4);
      CHECK((long long)s.groups * s.per_group >= nset);
      CHECK(s.total == (long long)items * s.groups);
    }
  CHECK(cfgmm::fock_share(1 << 25, 300, ctas).total == (1ll << 25) * 75);
  CHECK(cfgmm::fock_share(7000, 3, ctas).groups == 1);  // many items: one group
  CHECK(cfgmm::fock_share(275, 4, ctas).groups == 4);   // few: a group for each vector
  return 0;
}
