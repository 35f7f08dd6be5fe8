// fake_cuda.cpp -- the CUDA runtime functions that the library's objects call, with no
// GPU behind them: the host side of the library runs on the CPU, and drivers see what it
// asks of the runtime (see fake_cuda.h).  Linked in place of cudart.
#include "fake_cuda.h"

#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <thread>
#include <utility>

struct CUstream_st {
  int dev;
  bool work = false;   // launched or copied since the last wait
  bool busy = false;   // a long kernel runs
};
struct CUevent_st {
  CUstream_st* at = nullptr;
};

namespace fake {
int fail_async_alloc = 0;
int word_reads = 0;
int free_races = 0;
int long_device = -1;
int bad_launches = 0;
std::string last_bad;
bool record = false;
std::vector<std::pair<std::string, cudaStream_t>> launches;

namespace {
std::mutex mu;
std::condition_variable cv;
bool launched = false;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
std::set<CUstream_st*> streams;
CUstream_st* legacy[2] = {new CUstream_st{0}, new CUstream_st{1}};
std::set<void*> async_mem, pinned;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, int> granted;  // dynamic shared memory
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Config config;

CUstream_st* of(cudaStream_t s) { return s ? s : legacy[device]; }

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

void work(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  of(s)->work = true;
}

// waits for the long kernel of a stream, then nothing is in flight there
void wait(CUstream_st* s) {
  std::unique_lock<std::mutex> lk(mu);
  cv.wait(lk, [&] { return !s->busy; });
  s->work = false;
}

cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  std::lock_guard<std::mutex> lk(mu);
  const auto g = granted.find({device, f});
  const size_t most = std::max<size_t>(48 << 10, g == granted.end() ? 0 : size_t(g->second));
  const bool empty = !grid.x || !grid.y || !grid.z || !block.x;
  if (empty || grid.y > 65535 || grid.z > 65535 || smem > most) {
    ++bad_launches;
    last_bad = names[f];
    return ret(empty ? cudaErrorInvalidConfiguration : cudaErrorInvalidValue);
  }
  if (record) launches.emplace_back(names[f], stream);
  CUstream_st* s = of(stream);
  s->work = true;
  if (long_device == device) {
    s->busy = true;
    launched = true;
  }
  return cudaSuccess;
}
}  // namespace

void release() {
  std::lock_guard<std::mutex> lk(mu);
  long_device = -1;
  for (CUstream_st* s : streams) s->busy = false;
  for (CUstream_st* s : legacy) s->busy = false;
  cv.notify_all();
}

bool running() {
  std::lock_guard<std::mutex> lk(mu);
  return launched;
}
}  // namespace fake

using namespace fake;

extern "C" {

// ---- registration and launch ------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *static_cast<cudaStream_t*>(stream) = config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem,
                             cudaStream_t s) {
  return launch(f, grid, block, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
  std::lock_guard<std::mutex> lk(mu);
  granted[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 74;
  return cudaSuccess;
}

// ---- devices and errors -----------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  device = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
  *lo = 0;
  *hi = -1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) {
  *p = nullptr;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }
cudaError_t cudaDeviceSynchronize() {
  std::set<CUstream_st*> all;
  {
    std::lock_guard<std::mutex> lk(mu);
    all = streams;
  }
  for (CUstream_st* s : all)
    if (s->dev == device) wait(s);
  wait(legacy[device]);
  return cudaSuccess;
}
// no driver behind the runtime; a tensor map is filled with nothing
static int encode_nothing(...) { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long,
                                    cudaDriverEntryPointQueryResult* q) {
  *f = reinterpret_cast<void*>(&encode_nothing);
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

// ---- memory -----------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : ret(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  if (fail_async_alloc > 0 && --fail_async_alloc == 0) {
    *p = nullptr;
    return ret(cudaErrorMemoryAllocation);
  }
  const cudaError_t e = cudaMalloc(p, n);
  std::lock_guard<std::mutex> lk(mu);
  if (e == cudaSuccess) async_mem.insert(*p);
  return e;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> lk(mu);
  if (async_mem.erase(p)) {  // no wait is made for such memory
    bool flying = legacy[0]->work || legacy[1]->work;
    for (CUstream_st* s : streams) flying |= s->work;
    free_races += flying;
  }
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  std::lock_guard<std::mutex> lk(mu);
  async_mem.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  const cudaError_t e = cudaMalloc(p, n);
  std::lock_guard<std::mutex> lk(mu);
  pinned.insert(*p);
  return e;
}
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> lk(mu);
  pinned.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::lock_guard<std::mutex> lk(mu);
  a->type = pinned.count(const_cast<void*>(p)) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::memmove(d, s, n);
  work(st);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t st) {
  for (size_t r = 0; r < h; ++r)
    std::memmove(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
  work(st);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  std::memset(d, v, n);
  work(st);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind,
                                    cudaStream_t st) {
  work(st);
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) {
  ++word_reads;
  std::memset(d, 0, n);  // the error words: none
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = nullptr;
  return ret(cudaErrorInvalidSymbol);
}

// ---- streams, events, graphs --------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = new CUstream_st{device};
  std::lock_guard<std::mutex> lk(mu);
  streams.insert(*s);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) {
  return cudaStreamCreateWithFlags(s, f);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  streams.erase(s);
  delete s;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  wait(of(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  static char some;
  *e = reinterpret_cast<cudaGraphExec_t>(&some);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  work(s);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t f, void* p) {
  f(p);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = new CUevent_st;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  e->at = of(s);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::unique_lock<std::mutex> lk(mu);
  cv.wait(lk, [&] { return !e->at || !e->at->busy; });
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

}  // extern "C"
