// fock.cuh -- the Fock-build contraction on the per-block compacted AO lists.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace cfgmm {

// How the kernel shares out its work: the items (block tiles x row tiles) once for each
// of `groups` groups of up to `per_group` weight vectors (the last may be empty), `total`
// in all.  Items take kFockVectors vectors at most, and fewer where `ctas` CTAs would
// have under 8 items each to draw.  Vectors are many where items are few and the other
// way round, but both are the caller's: the product takes 64 bits.
constexpr int kFockVectors = 4;
struct FockShare {
  int groups, per_group;
  long long total;
};
__host__ __device__ inline FockShare fock_share(int items, int nset, int ctas) {
  // in 32 bits as far as that goes: a 64-bit division takes a small call's CTAs 0.1 us
  const unsigned least = (unsigned(nset) + kFockVectors - 1) / kFockVectors;
  const unsigned one = items > 0 ? items : 1;
  const unsigned wanted = (8u * ctas + one - 1) / one;
  const unsigned most = wanted < unsigned(nset) ? wanted : nset;
  FockShare s;
  s.groups = int(least > most ? least : most);
  s.per_group = int((unsigned(nset) + s.groups - 1) / s.groups);
  s.total = (long long)items * s.groups;
  return s;
}

// Device scratch (bytes) of fock_compact_fp64: active lists, work list, counters.
size_t fock_compact_workspace(size_t nao, size_t ngrid, size_t nset, size_t blk);

// vs[s*stride_ao^2 + u*stride_ao + v] += sum over g with tab[u][g/blk] and
// tab[v][g/blk] of ao_lhs[u][g] * ws[s*stride_grid + g] * ao_rhs[v][g], for
// s < nset, on `stream`; device pointers; `workspace` holds
// fock_compact_workspace(...) bytes, 256-byte aligned.
cudaError_t fock_compact_fp64(double* vs, const double* ws, const double* ao_lhs,
                              const double* ao_rhs, size_t stride_ao, size_t stride_grid,
                              int nao, int ngrid, int nset, const uint8_t* tab, size_t ldtab,
                              int blk, void* workspace, cudaStream_t stream);

// Sticky error word of the kernel's bounded waits (0 = none).
cudaError_t fock_reset_error(cudaStream_t stream);
cudaError_t fock_read_error(int* code);

}  // namespace cfgmm
