// The masked GEMM takes any BLKSIZE up to its limit just below 2^31, also one that added
// to n passes 2^31: one column block wider than C.
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t m = 300, n = 16384, k = 300;
  std::vector<double> c(m * n), a(m * k), b(k * n);
  std::vector<uint8_t> tab(k, 1);
  for (size_t blk : {size_t(20000), size_t(INT_MAX) - 16384, size_t(INT_MAX) - 4097,
                     size_t(INT_MAX) - 4096})
    for (int precision : {CFGMM_PREC_FP64, CFGMM_PREC_OZAKI_INT8}) {
      const int rc = cfgmm_matmul_non0tab_dev(c.data(), a.data(), b.data(), m, n, k, k, n, n, 0, 0,
                                              tab.data(), 1, blk, precision, nullptr);
      if (rc != CFGMM_OK) std::fprintf(stderr, "BLKSIZE %zu: %s\n", blk, fake::last_bad.c_str());
      CHECK(rc == CFGMM_OK);
    }
  return 0;
}
