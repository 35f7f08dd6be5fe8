// Which forms of the masked FP64 GEMM are enqueued: the compacted one, the dense one, or
// both with the device's choice between them; and a product whose aligned copies do not fit
// in memory runs without them.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

enum { kDense = 1, kCompacted = 2 };

int forms(size_t m, size_t n, size_t k, size_t blk, int transa, size_t pad) {
  const size_t lda = (transa ? m : k) + pad, ldb = n + pad, nblk = (n + blk - 1) / blk;
  std::vector<double> a((transa ? k : m) * lda), b(k * ldb), c(m * n);
  std::vector<uint8_t> tab(k * nblk, 1);
  fake::launches.clear();
  CHECK(cfgmm_matmul_non0tab_dev(c.data(), a.data(), b.data(), m, n, k, lda, ldb, n, transa, 0,
                                 tab.data(), nblk, blk, CFGMM_PREC_FP64, nullptr) == CFGMM_OK);
  int f = 0;
  for (const auto& l : fake::launches) {
    if (l.first.find("dgemm_mask_kernel") != std::string::npos) f |= kCompacted;
    if (l.first.find("12dgemm_kernel") != std::string::npos) f |= kDense;
  }
  return f;
}

int main() {
  fake::record = true;
  CHECK(forms(200, 900, 1000, 48, 0, 0) == kDense);       // up to 4e8 flops
  CHECK(forms(500, 2000, 500, 24, 0, 0) == kDense);       // blocks under 32 columns
  CHECK(forms(64, 16384, 500, 33, 0, 0) == kDense);       // the lists and copies alone cost more
  CHECK(forms(9, 16384, 1600, 48, 1, 1) == kDense);       // so do both operands' copies
  CHECK(forms(20000, 62, 500, 4096, 1, 0) == kCompacted);  // a block wider than C
  CHECK(forms(300, 2000, 1500, 48, 0, 0) == kCompacted);  // too small for both
  CHECK(forms(2228, 8000, 2228, 48, 0, 0) == kCompacted);
  CHECK(forms(2228, 8000, 2228, 33, 0, 0) == (kCompacted | kDense));  // 33 of 48 columns used
  CHECK(forms(130, 8000, 2228, 48, 1, 1) == (kCompacted | kDense));   // 130 of 256 rows used
  CHECK(forms(2228, 2000, 2228, 48, 0, 0) == (kCompacted | kDense));  // 5.1 rounds of items
  std::vector<double> x(2000 * 2001), y(2000 * 2001), z(2000 * 2000);
  for (int fail : {0, 1}) {
    fake::launches.clear();
    fake::fail_async_alloc = fail;
    CHECK(cfgmm_matmul_dev(z.data(), x.data(), y.data(), 2000, 2000, 2000, 2001, 2001, 2000, 0, 0,
                           CFGMM_PREC_FP64, nullptr) == CFGMM_OK);
    fake::fail_async_alloc = 0;
    CHECK(fake::launches.size() == (fail ? 1 : 3));
  }
  return 0;
}
