// A kernel's leave to use more than 48 KB of shared memory is each device's own: split
// contractions in the pair form, of so many tiles that the matching needs it, on one
// device after the other.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../include/cfgmm.h"
#include "fake_cuda.h"

int main() {
  const size_t nao = 1100, blk = 64;
  for (size_t tiles : {400, 4090}) {
    const size_t ngrid = tiles * blk;
    std::vector<double> rho(ngrid), ao(nao * ngrid), dms(nao * nao);
    std::vector<uint8_t> tab(nao * tiles, 1);
    for (int dev : {0, 1}) {
      cudaSetDevice(dev);
      const int rc = cfgmm_aodmao2rho_dev(rho.data(), dms.data(), ao.data(), ao.data(), nao, ngrid,
                                          nao, ngrid, 1, tab.data(), tiles, blk,
                                          CFGMM_PREC_OZAKI_INT8, nullptr);
      if (rc != CFGMM_OK) std::fprintf(stderr, "device %d: %s\n", dev, fake::last_bad.c_str());
      CHECK(rc == CFGMM_OK);
    }
  }
  return 0;
}
