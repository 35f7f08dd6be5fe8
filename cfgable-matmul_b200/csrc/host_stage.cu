// host_stage.cu -- copies between pageable host memory and the device (host_stage.cuh).
#include "host_stage.cuh"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

#if defined(__x86_64__)
#include <emmintrin.h>
#endif

namespace cfgmm {
namespace {

constexpr size_t kSlot = size_t(1) << 20;      // bytes of a pinned buffer
constexpr int kMaxWorkers = 6;  // copying threads, the caller among them
// Smaller copies go the driver's way.
constexpr size_t kDirectUp = size_t(1) << 20, kDirectDown = size_t(256) << 10;

// The driver takes 9 us for a piece, one after another, and a thread 80 us to fill 1 MB.
// A contiguous upload: four threads (six are no faster), two pieces or more for each.
constexpr int kUploadThreads = 4;
size_t upload_piece(size_t bytes) {
  const size_t each = bytes / (2 * kUploadThreads);
  return std::min(kSlot, std::max(size_t(256) << 10, (each + 4095) / 4096 * 4096));
}
// The present tiles of a table, whose packing takes longer than a plain copy: all threads,
// one piece for each where that fits, else four.  A density call with so many MB of tiles,
// us with 3, 4 and 6 threads: 5.6 928 635 581; 11.3 1195 989 840; 45.8 4391 3556 2888; 110
// 8575 7112 5889.
size_t tiles_piece(size_t bytes, int threads) {
  const size_t one = bytes / threads + bytes / (16 * threads);
  return one <= kSlot ? std::max(size_t(256) << 10, one)
                      : std::min(kSlot, std::max(size_t(512) << 10, bytes / (4 * threads)));
}
// A download: the caller alone below 1 MB, else four threads.  A product with so many MB of
// C, us with 1, 2, 4 and 6 threads: 0.7 202 256 281 284; 1.9 560 394 321 334; 7.6 1761 1179
// 698 772; 30 3750 2435 1841 1801.
int download_threads(size_t bytes) { return bytes < (size_t(1) << 20) ? 1 : 4; }
size_t download_piece(size_t bytes) {
  const size_t each = bytes / 12;
  return std::min(kSlot, std::max(size_t(128) << 10, (each + 4095) / 4096 * 4096));
}

// Copies into a pinned buffer past the caches (the piece ends with fill_done): the link's
// reads of lines that another core has just written go at a fifth of its speed, the more
// cores the slower, and the device waits for them.  us of a density call with so many MB of
// phi, a product's with three arrays: 2 threads through the caches, 4 of them, 4 past them:
// 3.8 365 522 222; 11.4 740 1004 470; 22.9 1235 1405 791; 3 x 3.7 934 755 730; 3 x 7.6 1734
// 1326 1078.  (The driver alone 315, 764, 1384; 1232, 2081.)
void fill(void* dst, const void* src, size_t n) {
#if defined(__x86_64__)
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  const size_t head = size_t(-reinterpret_cast<uintptr_t>(d)) & 15;
  if (n >= 64 + head) {
    std::memcpy(d, s, head);
    for (d += head, s += head, n -= head; n >= 64; d += 64, s += 64, n -= 64) {
      __m128i x[4];
      for (int i = 0; i < 4; ++i) x[i] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s) + i);
      for (int i = 0; i < 4; ++i) _mm_stream_si128(reinterpret_cast<__m128i*>(d) + i, x[i]);
    }
  }
  std::memcpy(d, s, n);
#else
  std::memcpy(dst, src, n);
#endif
}
void fill_done() {
#if defined(__x86_64__)
  _mm_sfence();
#endif
}

// A few threads that run one job at a time.  They live as long as the process: the
// object is never destroyed, so none of them meets a destroyed mutex at exit.
class Workers {
 public:
  static Workers& get() {
    static Workers* w = new Workers;
    return *w;
  }
  int count() const { return 1 + int(threads_); }
  // fn(worker) on up to `most` threads, worker 0 being the caller; returns when all are
  // done.  While another device's copy has the threads, on the caller alone, so that no
  // device waits for another.  (By address, without a std::function: nothing is allocated
  // that could fail.)
  template <class F>
  void run(F& fn, int most) {
    std::unique_lock<std::mutex> one(job_mu_, std::try_to_lock);
    const int helpers = std::min(most - 1, int(threads_));
    if (!one || helpers <= 0) return fn(0);
    {
      std::lock_guard<std::mutex> lk(mu_);
      call_ = [](void* f, int worker) { (*static_cast<F*>(f))(worker); };
      arg_ = &fn;
      running_ = helpers;
      for (int i = 1; i <= helpers; ++i) job_[i] = true;
    }
    for (int i = 1; i <= helpers; ++i) start_[i].notify_one();
    fn(0);
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [&] { return running_ == 0; });
  }

 private:
  Workers() {
    const unsigned hw = std::thread::hardware_concurrency();
    const int want = std::max(1, std::min(kMaxWorkers, int(hw / 2))) - 1;
    for (int i = 0; i < want; ++i) {
      try {
        std::thread([this, i] { loop(i + 1); }).detach();
      } catch (const std::system_error&) {
        break;  // fewer threads
      }
      ++threads_;
    }
  }
  void loop(int worker) {
    for (;;) {
      void (*call)(void*, int);
      void* arg;
      {
        std::unique_lock<std::mutex> lk(mu_);
        start_[worker].wait(lk, [&] { return job_[worker]; });
        job_[worker] = false;
        call = call_;
        arg = arg_;
      }
      call(arg, worker);
      std::lock_guard<std::mutex> lk(mu_);
      if (--running_ == 0) done_.notify_one();
    }
  }
  std::mutex job_mu_, mu_;
  std::condition_variable start_[kMaxWorkers], done_;
  bool job_[kMaxWorkers] = {};
  void (*call_)(void*, int) = nullptr;
  void* arg_ = nullptr;
  int running_ = 0;
  size_t threads_ = 0;
};

// A row's present tiles from `packed` (offsets[row] on, one after the other) to their
// places; CTA per row.
__global__ void __launch_bounds__(256)
spread_tiles(double* __restrict__ dst, size_t ld, const double* __restrict__ packed,
             const unsigned long long* __restrict__ offsets, const uint8_t* __restrict__ tab,
             size_t ldtab, long long cols, long long blk, int nblk) {
  __shared__ int warp_tot[8];
  __shared__ int list[256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* src = packed + offsets[blockIdx.x];
  double* row = dst + size_t(blockIdx.x) * ld;
  const uint8_t* t = tab + size_t(blockIdx.x) * ldtab;
  for (int b0 = 0; b0 < nblk; b0 += 256) {
    const int b = b0 + tid;
    const bool on = b < nblk && t[b] != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) warp_tot[warp] = __popc(bal);
    __syncthreads();
    int at = 0, total = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) at += warp_tot[w];
      total += warp_tot[w];
    }
    if (on) list[at + __popc(bal & ((1u << lane) - 1u))] = b;
    __syncthreads();
    const long long n = (long long)total * blk;
    for (long long i = tid; i < n; i += 256) {
      const long long q = i / blk, col = list[q] * blk + (i - q * blk);
      if (col < cols) row[col] = src[i];  // only the row's last tile can be short
    }
    src += n;
    __syncthreads();
  }
}

}  // namespace

bool host_pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t HostStage::ensure() try {
  const size_t slots = 2 * size_t(Workers::get().count());
  if (!pinned_) {
    const cudaError_t err =
        cudaHostAlloc(reinterpret_cast<void**>(&pinned_), slots * kSlot, cudaHostAllocPortable);
    if (err != cudaSuccess) {
      pinned_ = nullptr;
      return err;
    }
  }
  while (events_.size() < slots) {
    cudaEvent_t e;
    const cudaError_t err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (err != cudaSuccess) return err;
    events_.push_back(e);
  }
  return cudaSuccess;
} catch (const std::exception&) {  // no memory for the threads or the events
  return cudaErrorMemoryAllocation;
}

void HostStage::release() {
  for (cudaEvent_t e : events_) cudaEventDestroy(e);
  events_.clear();
  if (pinned_) cudaFreeHost(pinned_);
  pinned_ = nullptr;
}

namespace {

// Runs piece(i, slot) for i < n on up to `threads` copying threads, with the device current on
// each and a free pinned buffer; `piece` fills it and enqueues its copy on `stream`,
// behind which the buffer's event is recorded.
template <class P>
cudaError_t run_pieces(char* pinned, const std::vector<cudaEvent_t>& events, size_t n,
                       int threads, cudaStream_t stream, const P& piece) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::atomic<size_t> next{0};
  std::atomic<int> failed{0};
  auto copy = [&](int worker) {
    cudaError_t e = worker > 0 ? cudaSetDevice(dev) : cudaSuccess;
    for (int turn = 0; e == cudaSuccess && failed.load() == 0; turn ^= 1) {
      const size_t i = next.fetch_add(1);
      if (i >= n) break;
      const size_t slot = 2 * size_t(worker) + turn;
      e = cudaEventSynchronize(events[slot]);  // an event never recorded is complete
      if (e == cudaSuccess) e = piece(i, pinned + slot * kSlot);
      if (e == cudaSuccess) e = cudaEventRecord(events[slot], stream);
    }
    if (e != cudaSuccess) {
      int none = 0;
      failed.compare_exchange_strong(none, int(e));
    }
  };
  Workers::get().run(copy, threads);
  return cudaError_t(failed.load());
}

}  // namespace

cudaError_t HostStage::upload(void* dst, size_t dpitch, const void* src, size_t spitch,
                              size_t width, size_t rows, cudaStream_t stream) {
  if (rows > 1 && dpitch == width && spitch == width) {
    width *= rows;
    dpitch = spitch = width;
    rows = 1;
  }
  if (width * rows < kDirectUp || !host_pageable(src) || ensure() != cudaSuccess) {
    cudaGetLastError();
    return rows == 1 ? cudaMemcpyAsync(dst, src, width, cudaMemcpyHostToDevice, stream)
                     : cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows,
                                         cudaMemcpyHostToDevice, stream);
  }
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  const size_t most = upload_piece(width * rows);
  if (width > most) {  // parts of a row
    const size_t per_row = (width + most - 1) / most;
    return run_pieces(pinned_, events_, per_row * rows, kUploadThreads, stream, [&](size_t i, char* slot) {
      const size_t r = i / per_row, off = i % per_row * most;
      const size_t n = std::min(most, width - off);
      fill(slot, s + r * spitch + off, n);
      fill_done();
      return cudaMemcpyAsync(d + r * dpitch + off, slot, n, cudaMemcpyHostToDevice, stream);
    });
  }
  const size_t some = most / width;  // rows
  const size_t pieces = (rows + some - 1) / some;
  return run_pieces(pinned_, events_, pieces, kUploadThreads, stream, [&](size_t i, char* slot) {
    const size_t r0 = i * some, n = std::min(some, rows - r0);
    for (size_t r = 0; r < n; ++r) fill(slot + r * width, s + (r0 + r) * spitch, width);
    fill_done();
    return cudaMemcpy2DAsync(d + r0 * dpitch, dpitch, slot, width, width, n,
                             cudaMemcpyHostToDevice, stream);
  });
}

cudaError_t HostStage::download(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  if (bytes < kDirectDown || !host_pageable(dst) || ensure() != cudaSuccess) {
    cudaGetLastError();
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
  }
  // A thread copies a piece out of one of its buffers while the next piece arrives in
  // the other.  The caller requests its first two here and waits for the first, that is
  // for all earlier work on the stream, before it takes the threads.
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  const size_t most = download_piece(bytes), n = (bytes + most - 1) / most;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  auto request = [&](size_t i, size_t slot) {
    const size_t off = i * most;
    cudaError_t e = cudaMemcpyAsync(pinned_ + slot * kSlot, s + off, std::min(most, bytes - off),
                                    cudaMemcpyDeviceToHost, stream);
    return e == cudaSuccess ? cudaEventRecord(events_[slot], stream) : e;
  };
  const size_t first = std::min<size_t>(n, 2);
  for (size_t i = 0; err == cudaSuccess && i < first; ++i) err = request(i, i);
  if (err == cudaSuccess) err = cudaEventSynchronize(events_[0]);
  if (err != cudaSuccess) return err;
  std::atomic<size_t> next{first};
  std::atomic<int> failed{0};
  auto copy = [&](int worker) {
    cudaError_t e = worker > 0 ? cudaSetDevice(dev) : cudaSuccess;
    size_t held[2] = {n, n};  // the pieces in this thread's buffers
    for (size_t i = 0; worker == 0 && i < first; ++i) held[i] = i;
    bool more = true;
    for (int turn = 0; e == cudaSuccess && failed.load() == 0; turn ^= 1) {
      const size_t slot = 2 * size_t(worker) + turn;
      char* buf = pinned_ + slot * kSlot;
      if (held[turn] < n) {
        e = cudaEventSynchronize(events_[slot]);
        if (e != cudaSuccess) break;
        const size_t off = held[turn] * most;
        std::memcpy(d + off, buf, std::min(most, bytes - off));
        held[turn] = n;
      }
      const size_t i = more ? next.fetch_add(1) : n;
      if (i < n) {
        e = request(i, slot);
        held[turn] = i;
      } else {
        more = false;
        if (held[turn ^ 1] >= n) break;
      }
    }
    if (e != cudaSuccess) {
      int none = 0;
      failed.compare_exchange_strong(none, int(e));
    }
  };
  Workers::get().run(copy, download_threads(bytes));
  return cudaError_t(failed.load());
}

size_t HostStage::tiles_elems(size_t rows, size_t cols, const uint8_t* tab, size_t ldtab,
                              size_t blk, std::vector<unsigned long long>* offsets) {
  const size_t nblk = (cols + blk - 1) / blk;
  offsets->resize(rows);
  unsigned long long at = 0;
  for (size_t r = 0; r < rows; ++r) {
    (*offsets)[r] = at;
    const uint8_t* t = tab + r * ldtab;
    unsigned n = 0;
    for (size_t b = 0; b < nblk; ++b) n += t[b] != 0;
    at += (unsigned long long)n * blk;
    if (t[nblk - 1]) at -= nblk * blk - cols;  // the last tile may be short
  }
  return size_t(at);
}

cudaError_t HostStage::upload_tiles(double* dst, double* packed, unsigned long long* d_offsets,
                                    const double* src, size_t ld, size_t rows, size_t cols,
                                    const uint8_t* tab, const uint8_t* d_tab, size_t ldtab,
                                    size_t blk, const std::vector<unsigned long long>& offsets,
                                    size_t total, cudaStream_t stream) {
  cudaError_t err = ensure();
  if (err != cudaSuccess) return err;
  const size_t nblk = (cols + blk - 1) / blk;
  // pieces of at most a buffer: whole rows, or a part of the tiles of a long one
  struct Piece {
    size_t row, b, elems;
    unsigned long long at;
  };
  std::vector<Piece> pieces;
  const int threads = Workers::get().count();
  const size_t most = std::max(tiles_piece(total * 8, threads) / 8, blk);  // blk * 8 <= kSlot: the caller's
  for (size_t r = 0; r < rows; ++r) {
    const unsigned long long at = offsets[r];
    const size_t n = size_t((r + 1 < rows ? offsets[r + 1] : total) - at);
    if (n == 0) continue;
    if (n > most) {
      size_t done = 0;
      for (size_t b = 0; b < nblk; ++b)
        if (tab[r * ldtab + b]) {
          const size_t w = std::min(blk, cols - b * blk);
          if (done == 0 || pieces.back().elems + w > most) pieces.push_back({r, b, 0, at + done});
          pieces.back().elems += w;
          done += w;
        }
    } else if (pieces.empty() || pieces.back().elems + n > most) {
      pieces.push_back({r, 0, n, at});
    } else {
      pieces.back().elems += n;
    }
  }
  err = cudaMemcpyAsync(d_offsets, offsets.data(), rows * sizeof(unsigned long long),
                        cudaMemcpyHostToDevice, stream);
  if (err != cudaSuccess) return err;
  err = run_pieces(pinned_, events_, pieces.size(), threads, stream, [&](size_t i, char* slot) {
    const Piece& p = pieces[i];
    double* to = reinterpret_cast<double*>(slot);
    size_t left = p.elems, r = p.row, b = p.b;
    while (left > 0) {
      if (b == nblk) {
        ++r;
        b = 0;
        continue;
      }
      const uint8_t* t = tab + r * ldtab;
      if (!t[b]) {
        ++b;
        continue;
      }
      size_t n = 0;  // a run of present tiles
      const size_t c0 = b * blk;
      while (b < nblk && t[b] && n < left) {
        n += std::min(blk, cols - b * blk);
        ++b;
      }
      fill(to, src + r * ld + c0, n * 8);
      to += n;
      left -= n;
    }
    fill_done();
    return cudaMemcpyAsync(packed + p.at, slot, p.elems * 8, cudaMemcpyHostToDevice, stream);
  });
  if (err != cudaSuccess) return err;
  if (total == 0) return cudaSuccess;
  spread_tiles<<<unsigned(rows), 256, 0, stream>>>(dst, ld, packed, d_offsets, d_tab, ldtab,
                                                   (long long)cols, (long long)blk, int(nblk));
  return cudaGetLastError();
}

}  // namespace cfgmm
