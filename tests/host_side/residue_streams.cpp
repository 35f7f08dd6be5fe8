// Where the residues of a split product's operands are formed: of one operand by columns
// (clusters) and one by rows, the one by columns is on the caller's stream, which starts
// first, and the one by rows beside it.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t n = 300;
  std::vector<double> a(n * n), b(n * n), c(n * n);
  cudaStream_t s;
  cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  fake::record = true;
  for (int transa : {0, 1})
    for (int transb : {0, 1}) {
      fake::launches.clear();
      CHECK(cfgmm_matmul_dev(c.data(), a.data(), b.data(), n, n, n, n, n, n, transa, transb,
                             CFGMM_PREC_OZAKI_INT8, s) == CFGMM_OK);
      int cols = 0, rows = 0;
      for (const auto& l : fake::launches) {
        const bool by_cols = l.first.find("residues_cols") != std::string::npos;
        const bool by_rows = l.first.find("residues_rows") != std::string::npos;
        cols += by_cols;
        rows += by_rows;
        if (transa == transb && by_cols) CHECK(l.second == s);
        if (transa == transb && by_rows) CHECK(l.second != s);
      }
      CHECK(cols == transa + !transb && rows == !transa + transb);
    }
  return 0;
}
