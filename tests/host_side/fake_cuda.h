// fake_cuda.h -- what a driver sees of the CUDA runtime that fake_cuda.cpp stands in for.
#pragma once
#include <cstddef>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime_api.h>

namespace fake {

// Two devices.  Device memory is host memory, zeroed; copies and memsets are done at
// once; kernels do nothing.  Every launch, copy and memset is "in flight" on its stream
// until a call that waits for it.
extern int fail_async_alloc;  // the n-th cudaMallocAsync from now on fails (0: none)
extern int word_reads;        // cudaMemcpyFromSymbol: copies that the host waits for
extern int free_races;        // cudaFree of cudaMallocAsync memory with work in flight
// A kernel launched on a stream of this device (-1: none) runs until release() is called.
extern int long_device;
void release();
bool running();  // such a kernel has been launched
// Launches with an empty grid or more dynamic shared memory than the function was
// granted on the launching device return an error, as the runtime's do.
extern int bad_launches;
extern std::string last_bad;
// With `record`, every launch: the kernel's (mangled) name and its stream.
extern bool record;
extern std::vector<std::pair<std::string, cudaStream_t>> launches;

}  // namespace fake

#define CHECK(cond)                                                        \
  do {                                                                     \
    if (!(cond)) {                                                         \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);      \
      std::_Exit(1);                                                       \
    }                                                                      \
  } while (0)
