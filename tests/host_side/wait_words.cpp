// The error words of the bounded waits are read one blocking copy each: a host call reads
// at most five of them (there are seven), the check of the device all that can be set.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t n = 100, blk = 50, nblk = 2;
  std::vector<double> a(n * n), b(n * n), c(n * n), rho(n);
  std::vector<float> fa(n * n), fc(n * n);
  std::vector<uint8_t> tab(n * nblk, 1);
  auto reads = [](int rc) {
    CHECK(rc == CFGMM_OK);
    const int r = fake::word_reads;
    fake::word_reads = 0;
    return r;
  };
  const size_t l = n * n;
  for (int p : {CFGMM_PREC_FP64, CFGMM_PREC_OZAKI_INT8}) {
    CHECK(reads(cfgmm_matmul_ex(c.data(), l, a.data(), l, b.data(), l, n, n, n, n, n, n, 0, 0, p)) <= 5);
    CHECK(reads(cfgmm_matmul_f32(fc.data(), l, fa.data(), l, fa.data(), l, n, n, n, n, n, n, 0, 0,
                                 p)) <= 5);
    const int masked =
        reads(cfgmm_matmul_non0tab_ex(c.data(), l, a.data(), l, b.data(), l, n, n, n, n, n, n, 0, 0,
                                      tab.data(), tab.size(), nblk, blk, p));
    CHECK(masked == 5);  // its own word among them
    CHECK(reads(cfgmm_aodmao2rho_ex(rho.data(), n, a.data(), l, b.data(), l, b.data(), l, n, n, n,
                                    n, 1, tab.data(), tab.size(), nblk, blk, p)) <= 5);
  }
  CHECK(reads(cfgmm_aodm_fock(c.data(), l, rho.data(), n, b.data(), l, b.data(), l, n, n, n, n, 1,
                              tab.data(), tab.size(), nblk, blk)) == 5);
  CHECK(reads(cfgmm_device_check()) == 6);
  return 0;
}
