// dgemm_fp64.cu -- C += op(A) * op(B) in FP64 on the B200 FP64 tensor cores.
//
// Semantics follow MatmulLoops::matmul_loop_parallel_mnk_pack_a
// (src/impl_matmul.rs:155-231): row-major operands, opA(i,p) = transa ?
// a[p*lda+i] : a[i*lda+p], opB(p,j) = transb ? b[j*ldb+p] : b[p*ldb+j], and the
// product is ACCUMULATED into C (impl_matmul.rs:31-46).
//
// FP64 has no tcgen05 kind, so the math is the FP64 tensor-core MMA (DMMA,
// mma.sync m16n8k8 f64), fed from shared memory.  CTA = 64 x 64 of C, four warps
// of 32 x 32, K steps of 16 in a ring of three (cp.async), four CTAs per SM.
//   * Why small tiles, four to an SM: each CTA's barriers and copy latency are
//     hidden by the other three.  3000 x 3000 x 3000: 1.65 ms (32.8 TFLOP/s, 89 %
//     of the measured DMMA peak); one 128 x 128 CTA of eight warps per SM, staged
//     by TMA from operands packed K-contiguous, took 1.86 ms with its packing.
//   * Copies of 16 bytes where an operand's rows are 16-byte aligned, of 8 bytes
//     otherwise (any leading dimension and base): 8-byte copies cost 5 to 10 % of
//     the whole product, so a large product first copies an unaligned operand into
//     aligned rows (see pack_pays).
//   * Where the tiles leave SMs idle, a cluster of 2, 4 or 8 CTAs shares a tile:
//     each takes a part of K, and after a cluster barrier each adds its share of
//     the rows over the parts, in their order, through distributed shared memory
//     into C.  No workspace, no second kernel, deterministic (see choose_splits).
//     131 x 257 x 300: 83 -> 14 us (6 tiles of 128 x 128 ran ten serial K steps of
//     4.3 us; now 15 x 8 CTAs of two or three steps).
//   * No transposition: an operand whose rows run along k is staged as [row][k]
//     (16-byte slots XOR-swizzled), one whose rows run along m (n) as [k][row]
//     with a pitch of 66 doubles.  Both give lane (g, q) of a fragment load the
//     k pair 2q, 2q + 1 in k-slots q and q + 4, so A and B agree, and both are
//     free of bank conflicts (8 lanes of a phase meet 8 distinct 16-byte groups:
//     the pitch is 2 modulo 16 doubles; see swz_key).
//   * Tiles come in groups of 24 tile rows, so that the CTAs running together (592)
//     cover about 1536 x 1536 of C and share their rows of A and B in L2.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"
#include "dgemm_fp64.cuh"

namespace cfgmm {
namespace {

namespace cg = cooperative_groups;

constexpr int TILE = 64;      // of C
constexpr int TK = 16;        // K step
constexpr int STAGES = 3;
constexpr int THREADS = 128;
constexpr int GROUP = 24;     // tile rows of a group (see above)
constexpr int KP = TILE + 2;  // pitch of a [k][row] tile
constexpr int OP = TK * KP;   // doubles of one staged operand (the larger of both layouts)
constexpr int CP = TILE + 2;  // pitch of the partial tile exchanged in a cluster
constexpr size_t SMEM = size_t(STAGES) * 2 * OP * 8;
static_assert(size_t(TILE) * CP * 8 <= SMEM, "the partial tile fits the stages");

// A kernel of one of two forms that both are enqueued: it runs when the device
// word (the choice made earlier on the stream) is zero / nonzero as wanted.
struct Gate {
  const int* word;  // null: always runs
  int want;
  __device__ __forceinline__ bool closed() const { return word && (*word != 0) != (want != 0); }
};

template <class T>
struct GemmArgs {
  T* c;
  const double* a;
  const double* b;
  int m, n, k;
  size_t lda, ldb, ldc;
  const uint8_t* tab;  // masked GEMM: element (p, j) of B counts if tab[p*ldtab + j/blk]
  size_t ldtab;
  int blk;
  int tiles_m, tiles_n;
  bool avec, bvec;  // rows of A / B 16-byte aligned: copies of two elements
  int splits;  // CTAs of a cluster, each with a part of the K steps
  Gate gate;
};

// One thread's copies of an operand's K step: kKContig: x[r*ld + k] into
// S[r][k]; otherwise x[k*ld + r] into S[k][r].  With `vec` (rows 16-byte aligned)
// four copies of two adjacent elements, otherwise eight of one.
template <bool kKContig>
struct Copier {
  const double* src;   // this thread's first element of the operand's first K step
  size_t ld;
  int rows_left;       // rows of the operand from this thread's first row on
  int r, k0;           // its first row (of the tile) and k (of the step)
  bool vec;
  const uint8_t* tab;  // mask column of this thread's row, else null (vec is off)
  size_t ldtab;

  __device__ __forceinline__ void init(const double* x, size_t ld_, int row0, int rows, bool vec_,
                                       int tid) {
    ld = ld_;
    vec = vec_;
    tab = nullptr;
    if (kKContig) {
      k0 = vec ? 2 * (tid & 7) : tid & 15;
      r = vec ? tid >> 3 : tid >> 4;
      src = x + size_t(row0 + r) * ld + k0;
    } else {
      r = vec ? 2 * (tid & 31) : tid & 63;
      k0 = vec ? tid >> 5 : tid >> 6;
      src = x + size_t(k0) * ld + row0 + r;
    }
    rows_left = rows - row0 - r;
  }

  // K step starting at k = kt into S; k from kend on is zero
  __device__ __forceinline__ void issue(double* S, int kt, int kend) const {
    const int kl = kend - kt - k0;  // k left from this thread's first on
    if (kKContig) {
      const double* at = src + kt;
      if (vec) {
        const int bytes = kl >= 2 ? 16 : (kl == 1 ? 8 : 0);
#pragma unroll
        for (int i = 0; i < 4; ++i, at += 16 * ld)
          cp_async_16_n(S + swz<TK>(r + 16 * i, k0), at, 16 * i < rows_left ? bytes : 0);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i, at += 8 * ld)
          cp_async_8(S + swz<TK>(r + 8 * i, k0), at, kl > 0 && 8 * i < rows_left);
      }
    } else {
      const double* at = src + size_t(kt) * ld;
      if (vec) {
        const int bytes = rows_left >= 2 ? 16 : (rows_left == 1 ? 8 : 0);
#pragma unroll
        for (int i = 0; i < 4; ++i, at += 4 * ld)
          cp_async_16_n(S + (k0 + 4 * i) * KP + r, at, 4 * i < kl ? bytes : 0);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i, at += 2 * ld) {
          bool ok = rows_left > 0 && 2 * i < kl;
          if (tab && ok) ok = tab[size_t(kt + k0 + 2 * i) * ldtab] != 0;
          cp_async_8(S + (k0 + 2 * i) * KP + r, at, ok);
        }
      }
    }
  }
};

// T: the type of C; an f32 element is widened, added to and rounded once.
template <bool TA, bool TB, class T>
__global__ void __launch_bounds__(THREADS, 4)
dgemm_kernel(const __grid_constant__ GemmArgs<T> p) {
  if (p.gate.closed()) return;  // every CTA of the grid alike
  extern __shared__ __align__(128) double gemm_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int g = lane >> 2, q = lane & 3;
  const int tile = blockIdx.x / p.splits, part = blockIdx.x % p.splits;
  const int per_group = GROUP * p.tiles_n;
  const int first = tile / per_group * GROUP, in_group = tile % per_group;
  const int rows_g = min(GROUP, p.tiles_m - first);
  const int m0 = (first + in_group % rows_g) * TILE, n0 = in_group / rows_g * TILE;
  const int steps = (p.k + TK - 1) / TK;
  const int s0 = int((long long)part * steps / p.splits);
  const int s1 = int((long long)(part + 1) * steps / p.splits);

  Copier<!TA> ca;
  Copier<TB> cb;
  ca.init(p.a, p.lda, m0, p.m, p.avec, tid);
  cb.init(p.b, p.ldb, n0, p.n, p.bvec, tid);
  if (!TB && p.tab && cb.rows_left > 0) {
    cb.tab = p.tab + (n0 + cb.r) / p.blk;
    cb.ldtab = p.ldtab;
  }
  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s0 + s < s1) {
      double* S = gemm_smem + s * 2 * OP;
      ca.issue(S, (s0 + s) * TK, p.k);
      cb.issue(S + OP, (s0 + s) * TK, p.k);
    }
    cp_async_commit();
  }
  for (int st = s0; st < s1; ++st) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    const int nx = st + STAGES - 1;
    if (nx < s1) {
      double* S = gemm_smem + ((nx - s0) % STAGES) * 2 * OP;
      ca.issue(S, nx * TK, p.k);
      cb.issue(S + OP, nx * TK, p.k);
    }
    cp_async_commit();
    const double* As = gemm_smem + ((st - s0) % STAGES) * 2 * OP;
    const double* Bs = As + OP;
#pragma unroll
    for (int kk = 0; kk < TK; kk += 8) {
      double2 a0[2], a1[2], b0[4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const int r = wm * 32 + mt * 16;
        if (TA) {  // k rows 2q, 2q + 1; rows 2g, 2g + 1 of the 16
          a0[mt] = *reinterpret_cast<const double2*>(As + (kk + 2 * q) * KP + r + 2 * g);
          a1[mt] = *reinterpret_cast<const double2*>(As + (kk + 2 * q + 1) * KP + r + 2 * g);
        } else {
          a0[mt] = *reinterpret_cast<const double2*>(As + swz<TK>(r + g, kk + 2 * q));
          a1[mt] = *reinterpret_cast<const double2*>(As + swz<TK>(r + g + 8, kk + 2 * q));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (TB)
          b0[j] = *reinterpret_cast<const double2*>(Bs + swz<TK>(wn * 32 + j * 8 + g, kk + 2 * q));
        else  // b0[2j'], b0[2j' + 1]: k rows 2q, 2q + 1; columns 2g, 2g + 1 of 16
          b0[j] = *reinterpret_cast<const double2*>(Bs + (kk + 2 * q + (j & 1)) * KP + wn * 32 +
                                                    (j >> 1) * 16 + 2 * g);
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double x0 = a0[mt].x, x1 = TA ? a0[mt].y : a1[mt].x;
          const double x2 = TA ? a1[mt].x : a0[mt].y, x3 = a1[mt].y;
          const double y0 = TB ? b0[j].x : (j & 1 ? b0[j & ~1].y : b0[j & ~1].x);
          const double y1 = TB ? b0[j].y : (j & 1 ? b0[j | 1].y : b0[j | 1].x);
          dmma_16x8x8(acc[mt][j], x0, x1, x2, x3, y0, y1);
        }
    }
  }
  cp_async_wait<0>();

  // accumulator (mt, j, 2h + e): this row and column of the tile
  auto row_of = [&](int mt, int h) { return wm * 32 + mt * 16 + (TA ? 2 * g + h : g + 8 * h); };
  auto col_of = [&](int j, int e) {
    return wn * 32 + (TB ? j * 8 + 2 * q + e : (j >> 1) * 16 + 4 * q + 2 * e + (j & 1));
  };
  if (p.splits == 1) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = m0 + row_of(mt, h);
        if (row >= p.m) continue;
        T* crow = p.c + size_t(row) * p.ldc + n0;
        double old[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            old[j][e] = n0 + col_of(j, e) < p.n ? double(crow[col_of(j, e)]) : 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (n0 + col_of(j, e) < p.n) crow[col_of(j, e)] = T(old[j][e] + acc[mt][j][2 * h + e]);
      }
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads();  // the stages are read
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          gemm_smem[row_of(mt, h) * CP + col_of(j, e)] = acc[mt][j][2 * h + e];
  cluster.sync();
  // each CTA adds its rows over the parts, in their order; a thread's reads of the
  // other CTAs' memory are all under way at once (in a loop over the parts, one after
  // another, whose registers also spilled in the main loop: 1000^3 91 -> 87 us, 3000 x 3000 x 300 196
  // -> 185, 3000^3 1.669 -> 1.648 ms; calls of a few tiles are bound by their launch)
  const int rows = TILE / p.splits;
  double v[2][8];
#pragma unroll 1
  for (int i0 = 0; i0 < rows * TILE / THREADS; i0 += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = (i0 + u) * THREADS + tid;
      const int r = part * rows + i / TILE, cc = i % TILE;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        v[u][s] = s < p.splits ? *cluster.map_shared_rank(gemm_smem + r * CP + cc, s) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = (i0 + u) * THREADS + tid;
      const int r = part * rows + i / TILE, cc = i % TILE;
      double sum = 0.0;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < p.splits) sum += v[u][s];
      if (m0 + r >= p.m || n0 + cc >= p.n) continue;
      T* dst = p.c + size_t(m0 + r) * p.ldc + n0 + cc;
      *dst = T(double(*dst) + sum);
    }
  }
  cluster.sync();  // a CTA's partial tile is read until here
}

// dst[r*pitch + c] = src[r*ld + c] (c < cols; with a mask, zero unless
// tab[r*ldtab + c/blk]): an operand into doubles in rows of an even pitch.  1024
// columns of a row per pass of a CTA.
template <class T>
__global__ void __launch_bounds__(256)
pack_aligned(double* __restrict__ dst, int pitch, const T* __restrict__ src, size_t ld,
             int rows, int cols, const uint8_t* __restrict__ tab, size_t ldtab, int blk,
             Gate gate) {
  if (gate.closed()) return;
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const T* s = src + size_t(r) * ld;
    double* d = dst + size_t(r) * pitch;
    double2 v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = blockIdx.x * 1024 + 512 * i + 2 * threadIdx.x;
      v[i].x = c < cols && (!tab || tab[size_t(r) * ldtab + c / blk]) ? double(s[c]) : 0.0;
      v[i].y = c + 1 < cols && (!tab || tab[size_t(r) * ldtab + (c + 1) / blk]) ? double(s[c + 1])
                                                                                : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = blockIdx.x * 1024 + 512 * i + 2 * threadIdx.x;
      if (c < pitch) *reinterpret_cast<double2*>(d + c) = v[i];
    }
  }
}

// dst[r][kk] = src[r * ld + kk] (kk < k), 0 for k <= kk < kpad: rows of a
// K-contiguous operand.  A warp per row, 256 columns per block.
__global__ void __launch_bounds__(256)
pack_rows(double* __restrict__ dst, const double* __restrict__ src, size_t ld, int rows, int k,
          int kpad, Gate gate) {
  if (gate.closed()) return;
  const int r = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (r >= rows) return;
  const double* srow = src + size_t(r) * ld;
  double* drow = dst + size_t(r) * kpad;
  for (int j = threadIdx.x & 31; j < 256; j += 32) {
    const int kk = blockIdx.x * 256 + j;
    if (kk < kpad) drow[kk] = kk < k ? srow[kk] : 0.0;
  }
}

// dst[j][p] = src[p * ld + j] for p < k (0 for k <= p < kpad), j < cols: the
// transpose into a K-contiguous operand, through a 32 x 32 shared tile.
__global__ void __launch_bounds__(256)
pack_transpose(double* __restrict__ dst, const double* __restrict__ src, size_t ld, int cols,
               int k, int kpad, Gate gate) {
  if (gate.closed()) return;
  __shared__ double t[32][33];
  const int j0 = blockIdx.x * 32, p0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const int p = p0 + ty + i, j = j0 + tx;
    t[ty + i][tx] = p < k && j < cols ? src[size_t(p) * ld + j] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const int j = j0 + ty + i, p = p0 + tx;
    if (j < cols && p < kpad) dst[size_t(j) * kpad + p] = t[tx][ty + i];
  }
}

template <bool TA, bool TB, class T>
cudaError_t launch_t(const GemmArgs<T>& p, cudaStream_t stream) {
  auto kern = dgemm_kernel<TA, TB, T>;
  cudaError_t err =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SMEM));
  if (err != cudaSuccess) return err;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(p.tiles_m) * p.tiles_n * p.splits);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = unsigned(p.splits);
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

// CTAs per tile.  An SM's time is taken as its CTAs times the K steps of each plus
// two for a CTA's start and end; its CTAs are counted between the most that an SM
// gets and the mean (they do not all start together), half a one more for the last
// to end, and at least 3 (fewer do not fill an SM).  The least time wins, the fewer
// parts of equals.  On 70 shapes (tiles 4 to 2500, k 100 to 6500) timed with 1, 2, 4
// and 8 parts the choice is within 0.8 % of the fastest on average and 9 % at worst;
// 130 x 130 x 5000 takes 269, 146, 75, 42 us with 1, 2, 4, 8 parts, 1200 x 1500 x 1000
// 166, 154, 142, 148, 2000 x 2000 x 500 146, 160, 176, 204.
struct Splits {
  int count;
  double time;  // the model's, in units of 0.56 us
};
Splits choose_splits(long long tiles, int steps, int nsm) {
  Splits best{1, 0.0};
  for (int s = 1; s <= 8 && (s == 1 || steps >= 2 * s); s *= 2) {
    const double mean = double(tiles * s) / nsm, most = double((tiles * s + nsm - 1) / nsm);
    const double t = std::max(0.5 * (most + mean) + 0.5, 3.0) * (double(steps) / s + 2.0);
    if (s == 1 || t < best.time) best = Splits{s, t};
  }
  return best;
}

bool al16(const void* x, size_t ld) {
  return (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ld % 2 == 0;
}

// CFGMM_DGEMM_PACK_MIN_FLOPS: products of at least so many flops copy unaligned
// operands (< 0: none does); without it the rule below.
double pack_min_flops() {
  static const double v = [] {
    const char* e = std::getenv("CFGMM_DGEMM_PACK_MIN_FLOPS");
    return e ? std::atof(e) : 0.0;
  }();
  return v;
}

// Whether to copy an unaligned operand of `elems` elements into aligned rows: its
// 8-byte copies cost about 4.5 % of the product at 32 TFLOP/s, the pass 16 bytes
// per element at 5.5 TB/s and a launch of 4 us.
bool pack_pays(int m, int n, int k, double elems) {
  const double flops = 2.0 * m * n * k, min = pack_min_flops();
  if (min != 0.0) return min > 0.0 && flops >= min;
  return 0.045 * flops / 32e12 > elems * 16.0 / 5.5e12 + 4e-6;
}

// f32 operands are widened into aligned rows of doubles, whatever their size, and the
// kernel adds to the f32 C itself (64-bit sums, one rounding).  Widening A, B and C
// and narrowing C in passes of their own: 390 x 200 x 1109 202 -> 34 us (K parts
// included), 691 x 2668 x 124 72 -> 60, 3448 x 3968 x 840 1008 -> 757.
template <class T>
cudaError_t gemm(T* c, const T* a, const T* b, int m, int n, int k, size_t lda, size_t ldb,
                 size_t ldc, bool transa, bool transb, const uint8_t* tab,
                 size_t ldtab, int blk, Gate gate, cudaStream_t stream) {
  const long long tiles_m = (m + TILE - 1) / TILE, tiles_n = (n + TILE - 1) / TILE;
  if (tiles_m * tiles_n > (1ll << 27)) return cudaErrorInvalidConfiguration;
  int dev = 0, nsm = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess)
    err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (err != cudaSuccess) return err;
  GemmArgs<T> p{};
  p.c = c;
  p.m = m;
  p.n = n;
  p.k = k;
  p.ldc = ldc;
  p.tiles_m = int(tiles_m);
  p.tiles_n = int(tiles_n);
  p.splits = choose_splits(tiles_m * tiles_n, (k + TK - 1) / TK, nsm).count;
  p.gate = gate;
  const int ar = transa ? k : m, ac = transa ? m : k, br = transb ? n : k, bc = transb ? k : n;
  constexpr bool widen = !std::is_same<T, double>::value;
  bool pa = widen || (!al16(a, lda) && pack_pays(m, n, k, double(m) * k));
  bool pb = widen || ((tab || !al16(b, ldb)) && pack_pays(m, n, k, double(n) * k));
  const int apitch = (ac + 1) / 2 * 2, bpitch = (bc + 1) / 2 * 2;
  const double *da = nullptr, *db = nullptr;
  if constexpr (!widen) {
    da = a;
    db = b;
  }
  double* ws = nullptr;
  if (pa || pb) {
    const size_t an = pa ? size_t(ar) * apitch : 0, bn = pb ? size_t(br) * bpitch : 0;
    err = cudaMallocAsync(reinterpret_cast<void**>(&ws), (an + bn) * 8, stream);
    if (err == cudaErrorMemoryAllocation && !widen) {  // it runs without the copies too
      cudaGetLastError();
      err = cudaSuccess;
      ws = nullptr;
      pa = pb = false;
    }
    if (err != cudaSuccess) return err;
    auto grid = [&](int pitch, int rows) {  // gated: few CTAs, soon over if they do not run
      const int across = (pitch + 1023) / 1024;
      return dim3(across, std::min(rows, gate.word ? 1024 / across + 1 : 65535));
    };
    if (pa) {
      pack_aligned<<<grid(apitch, ar), 256, 0, stream>>>(
          ws, apitch, a, lda, ar, ac, nullptr, 0, 1, gate);
      da = ws;
      lda = apitch;
    }
    if (pb) {
      pack_aligned<<<grid(bpitch, br), 256, 0, stream>>>(
          ws + an, bpitch, b, ldb, br, bc, tab, ldtab, blk, gate);
      db = ws + an;
      ldb = bpitch;
      tab = nullptr;
    }
    err = cudaGetLastError();
  }
  p.a = da;
  p.b = db;
  p.lda = lda;
  p.ldb = ldb;
  p.tab = tab;
  p.ldtab = ldtab;
  p.blk = blk;
  p.avec = al16(da, lda);
  p.bvec = !tab && al16(db, ldb);
  if (err == cudaSuccess) {
    if (!transa)
      err = transb ? launch_t<false, true>(p, stream) : launch_t<false, false>(p, stream);
    else
      err = transb ? launch_t<true, true>(p, stream) : launch_t<true, false>(p, stream);
  }
  if (ws) {
    const cudaError_t e2 = cudaFreeAsync(ws, stream);
    if (err == cudaSuccess) err = e2;
  }
  return err;
}

// The dense form of a masked product (in-place copies of B ask for the mask 8 bytes at a
// time): the model of choose_splits and the copies, 0.95 to 1.12 of what eight in ten of 22
// shapes of 50 us to 5 ms take, 0.90 to 1.21 of all.
double masked_dense_us(int m, int n, int k, bool transa) {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      nsm <= 0) {
    cudaGetLastError();
    nsm = 148;
  }
  const long long tiles = (long long)((m + TILE - 1) / TILE) * ((n + TILE - 1) / TILE);
  const double us = 0.56 * choose_splits(tiles, (k + TK - 1) / TK, nsm).time;
  if (pack_pays(m, n, k, double(n) * k)) return 1.03 * us + 16.0 * n * k / 5.5e6 + 6.0;
  return (transa ? 1.4 : 1.28) * us + 12.0;
}

}  // namespace

cudaError_t dgemm_fp64(double* c, const double* a, const double* b, int m, int n, int k,
                       size_t lda, size_t ldb, size_t ldc, bool transa, bool transb,
                       cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  return gemm(c, a, b, m, n, k, lda, ldb, ldc, transa, transb, nullptr, 0, 1, Gate{nullptr, 0},
              stream);
}

cudaError_t dgemm_f32(float* c, const float* a, const float* b, int m, int n, int k, size_t lda,
                      size_t ldb, size_t ldc, bool transa, bool transb, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  return gemm(c, a, b, m, n, k, lda, ldb, ldc, transa, transb, nullptr, 0, 1, Gate{nullptr, 0},
              stream);
}

cudaError_t dgemm_pack_kmajor(double* dst, const double* a, size_t lda, int m, int k, int pitch,
                              bool transa, const int* run, cudaStream_t stream) {
  const Gate gate{run, 1};
  if (transa)
    pack_rows<<<dim3((pitch + 255) / 256, (k + 7) / 8), 256, 0, stream>>>(dst, a, lda, k, m, pitch,
                                                                         gate);
  else
    pack_transpose<<<dim3((k + 31) / 32, (pitch + 31) / 32), 256, 0, stream>>>(
        dst, a, lda, k, m, pitch, gate);
  return cudaGetLastError();
}

cudaError_t dgemm_fp64_non0tab(double* c, const double* a, const double* b, int m, int n, int k,
                               size_t lda, size_t ldb, size_t ldc, bool transa,
                               const uint8_t* tab, size_t ldtab, int blk, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  if (!dgemm_mask_applies(m, n, k, blk))
    return gemm(c, a, b, m, n, k, lda, ldb, ldc, transa, false, tab, ldtab, blk, Gate{nullptr, 0},
                stream);
  // Where the dense form can be the faster one, both are enqueued and the device picks by
  // the share of present tiles: the host does not know it without waiting for the mask.
  // The second form's launches cost 3 to 10 us, so not for smaller products (of the dense
  // form's padded rows): at 0.05 present 84 -> 95 us at 2228 x 2000 x 2228, with all tiles
  // present 821 -> 704.  Where the lists and copies leave the compacted form no gain above
  // a share of 0.15, the dense one runs alone (64 x 16384 x 500, BLKSIZE 33, 0.3 present: 93
  // -> 59 us).
  const double dense = masked_dense_us(m, n, k, transa);
  const MaskTimes t = dgemm_mask_times(a, b, m, n, k, lda, ldb, transa, blk);
  if (dense <= t.lists + t.copies + 0.15 * t.products)
    return gemm(c, a, b, m, n, k, lda, ldb, ldc, transa, false, tab, ldtab, blk, Gate{nullptr, 0},
                stream);
  const double rows = (m + TILE - 1) / TILE * double(TILE);
  double share = (dense - t.copies) / t.products;  // up to which the compacted form is faster
  if (2.0 * rows * n * k < 2e9) share = 1.0;
  const size_t wsb = dgemm_mask_workspace(a, b, m, n, k, lda, ldb, transa, blk);
  int* compact = nullptr;  // the choice, outliving the compacted form's scratch
  void* ws = nullptr;
  cudaError_t err = cudaSuccess;
  if (share < 1.0) {
    if ((err = cudaMallocAsync(reinterpret_cast<void**>(&compact), 256, stream)) != cudaSuccess)
      return err;
    err = cudaMallocAsync(&ws, wsb, stream);
  } else {
    err = cudaMallocAsync(&ws, wsb + 256, stream);
  }
  if (err == cudaSuccess) {
    err = dgemm_mask_compact(
        c, a, b, m, n, k, lda, ldb, ldc, transa, tab, ldtab, blk, share,
        compact ? compact : reinterpret_cast<int*>(static_cast<char*>(ws) + wsb), ws, stream);
    const cudaError_t e2 = cudaFreeAsync(ws, stream);
    if (err == cudaSuccess) err = e2;
  }
  if (compact) {
    if (err == cudaSuccess)
      err = gemm(c, a, b, m, n, k, lda, ldb, ldc, transa, false, tab, ldtab, blk,
                 Gate{compact, 0}, stream);
    const cudaError_t e3 = cudaFreeAsync(compact, stream);
    if (err == cudaSuccess) err = e3;
  }
  return err;
}

}  // namespace cfgmm
