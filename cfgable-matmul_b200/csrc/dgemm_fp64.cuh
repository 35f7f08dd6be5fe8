// dgemm_fp64.cuh -- internal launcher of the FP64 tensor-core DGEMM.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cfgmm {

// C[i*ldc+j] += sum_p opA(i,p) opB(p,j) on `stream`; device pointers.
cudaError_t dgemm_fp64(double* c, const double* a, const double* b, int m, int n, int k,
                       size_t lda, size_t ldb, size_t ldc, bool transa, bool transb,
                       cudaStream_t stream);

// The same on f32 data: operands widened exactly, FP64 arithmetic, each element of C
// rounded once.
cudaError_t dgemm_f32(float* c, const float* a, const float* b, int m, int n, int k, size_t lda,
                      size_t ldb, size_t ldc, bool transa, bool transb, cudaStream_t stream);

// Masked GEMM (src/impl_matmul_non0tab.rs:210-306): B is not transposed;
// element (p, j) of B takes part only when tab[p * ldtab + j / blk] != 0.
cudaError_t dgemm_fp64_non0tab(double* c, const double* a, const double* b, int m, int n, int k,
                               size_t lda, size_t ldb, size_t ldc, bool transa,
                               const uint8_t* tab, size_t ldtab, int blk, cudaStream_t stream);

// The masked GEMM on each column block's compacted rows (dgemm_mask.cu).
// dgemm_mask_applies: the shapes it takes; dgemm_mask_times: what it takes, in us (its
// products with every tile present).  dgemm_mask_compact enqueues the lists, the choice and the kernel: where more
// than max_share (< 1) of the tiles is present nothing is added to C and the
// device word *compact is 0 (the caller then enqueues the dense form gated on
// it), otherwise it is 1.
bool dgemm_mask_applies(int m, int n, int k, int blk);
struct MaskTimes {
  double lists, copies, products;
};
MaskTimes dgemm_mask_times(const double* a, const double* b, int m, int n, int k, size_t lda,
                           size_t ldb, bool transa, int blk);
size_t dgemm_mask_workspace(const double* a, const double* b, int m, int n, int k, size_t lda,
                            size_t ldb, bool transa, int blk);
cudaError_t dgemm_mask_compact(double* c, const double* a, const double* b, int m, int n, int k,
                               size_t lda, size_t ldb, size_t ldc, bool transa,
                               const uint8_t* tab, size_t ldtab, int blk, double max_share,
                               int* compact, void* workspace, cudaStream_t stream);
// Sticky error word of the compacted form's bounded waits (0 = none).
cudaError_t dgemm_mask_reset_error(cudaStream_t stream);
cudaError_t dgemm_mask_read_error(int* code);

// dst[p*pitch + i] = opA(i, p) for p < k, i < m, 0 for m <= i < pitch; with
// `run`, only when *run != 0 on the device.
cudaError_t dgemm_pack_kmajor(double* dst, const double* a, size_t lda, int m, int k, int pitch,
                              bool transa, const int* run, cudaStream_t stream);

// Fock-build contraction of one density set on `stream`: V[u*ldv + v] +=
// sum over g with tab[u][g/blk] and tab[v][g/blk] of ao_lhs[u][g] w[g]
// ao_rhs[v][g].  `workspace` holds fock_fp64_workspace(nao, ngrid) bytes,
// 256-byte aligned; pack_rhs = false reuses the right operand and activity map
// left there by a previous call with the same ao_rhs and mask.
size_t fock_fp64_workspace(int nao, int ngrid);
cudaError_t fock_fp64(double* v, size_t ldv, const double* w, const double* ao_lhs,
                      const double* ao_rhs, size_t stride_grid, int nao, int ngrid,
                      const uint8_t* tab, size_t ldtab, int blk, bool pack_rhs, void* workspace,
                      cudaStream_t stream);

// Sticky error word of the dense Fock form's bounded waits (0 = none).
cudaError_t fock_dense_reset_error(cudaStream_t stream);
cudaError_t fock_dense_read_error(int* code);

}  // namespace cfgmm
