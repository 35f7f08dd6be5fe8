// host_stage.cuh -- copies between pageable host memory and the device.
//
// cudaMemcpyAsync from pageable memory goes through one driver thread's copies into
// its own pinned buffers (10 GB/s here, 19 when the source is in the caches; the link
// takes 55).  A HostStage has pinned buffers of its own, which several threads fill (or
// empty) at once while the copies of the buffers filled before are on the link.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace cfgmm {

// Whether `p` is host memory that CUDA does not know (neither pinned nor managed).
bool host_pageable(const void* p);

// One device's buffers.  Calls are made with that device current and are not
// concurrent with one another (the device state's lock).  The copying threads serve
// one device at a time; a call that finds them taken copies by itself.
class HostStage {
 public:
  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;

  // cudaMemcpy2DAsync host -> device / device -> host on `stream`.  From pageable
  // memory (and enough of it) through the buffers: an upload returns when `src` has
  // been read, a download when `dst` has been written.
  cudaError_t upload(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                     size_t rows, cudaStream_t stream);
  cudaError_t upload(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    return upload(dst, bytes, src, bytes, bytes, 1, stream);
  }
  cudaError_t download(void* dst, const void* src, size_t bytes, cudaStream_t stream);

  // The present tiles of a table (rows x cols doubles at pitch ld; tile (r, b) =
  // columns b blk .. of row r, present if tab[r ldtab + b]) to the device, packed
  // into `packed` and spread from there into `dst` at the same pitch.  Elements of
  // absent tiles are neither read nor written.  tiles_elems: the elements of the
  // present tiles, i.e. the doubles that `packed` holds; offsets[r]: those before
  // row r (`d_offsets`: rows words of device scratch).
  static size_t tiles_elems(size_t rows, size_t cols, const uint8_t* tab, size_t ldtab, size_t blk,
                            std::vector<unsigned long long>* offsets);
  cudaError_t upload_tiles(double* dst, double* packed, unsigned long long* d_offsets,
                           const double* src, size_t ld, size_t rows, size_t cols,
                           const uint8_t* tab, const uint8_t* d_tab, size_t ldtab, size_t blk,
                           const std::vector<unsigned long long>& offsets, size_t total,
                           cudaStream_t stream);

  // Frees the buffers (no copy may be in flight).
  void release();

 private:
  cudaError_t ensure();
  char* pinned_ = nullptr;
  std::vector<cudaEvent_t> events_;  // two per copying thread
};

}  // namespace cfgmm
