// dgemm_mask.cu -- the masked GEMM on the compacted rows of each column block:
//
//   C[i][j] += sum_{p in I(b)} opA(i,p) B[p][j],  b = j / BLK,
//   I(b) = { p < k : tab[p*ldtab + b] != 0 } in ascending order
//
// (matmul_loop_parallel_mnk_pack_a_non0tab, src/impl_matmul_non0tab.rs:210-306;
// the lists are the reference's get_indices_from_non0tab, :118-129).  Only the
// products of present tiles are formed; rows p outside I(b) are not read.
//
// Operands are "k-major": row p of A^T (opA(0..m-1, p), contiguous) and row p of
// B.  A^T is A itself when transa and its rows are 16-byte aligned, else one
// packed copy; B is used in place when every (row, block) piece starts on a
// 16-byte boundary, else its present tiles are copied once into aligned rows.
//
// Measured at 2228 x 16384 x 2228, BLKSIZE 48, 30 % of the tiles present: 1.60 ms
// (30.5 TFLOP/s of present products; the floor at the DMMA peak of 37 is 1.32),
// where the dense form takes 5.04 ms; every tile present: 5.11 against 5.06 ms.
//
// dgemm_mask_kernel: work item = (column block piece of up to 64 columns, 128
// rows of C).  One producer warp fetches 16 list rows per stage with untiled
// bulk copies (one per row: 128 doubles of A^T, the piece's columns of B), eight
// consumer warps (16 rows x all columns each) run DMMA m16n8k8 and add into C.
//   * Why compaction and not zero-filled B: the FP64 tensor pipe bounds both
//     forms, and the dense one issues 1/density times the products.
//   * Why two CTAs per SM: while one adds its tile into C (or starts an item)
//     the other keeps the tensor pipe busy.
//   * Row pitches of 128 + 4 and W + 4 doubles: a quarter warp's 16-byte
//     fragment loads (k rows q = 0..3, adjacent column pairs g, g + 1) meet 8
//     distinct 16-byte bank groups, because the pitch is 2 modulo 8 of them.
//     A lane's pair of adjacent rows (columns) is used as rows g and g + 8 of
//     one m16 tile (as the same column of two n8 tiles): a permutation of C's
//     rows and columns that the epilogue undoes.
#include <algorithm>

#include "aodmao2rho_fp64.cuh"
#include "common.cuh"
#include "dgemm_fp64.cuh"
#include "tcgen05.cuh"

namespace cfgmm {
namespace {

__device__ int g_mask_error;

constexpr int TM = 128;      // rows of C per item
constexpr int TK = 16;       // list rows per stage
constexpr int STAGES = 4;
constexpr int CONS = 8;      // consumer warps, 16 rows each
constexpr int THREADS = 32 * (CONS + 1);
constexpr int PA = TM + 4;   // A row pitch in shared memory (doubles)
constexpr int MAXW = 64;     // columns per item at most

template <int NTP>
constexpr int stage_doubles() { return TK * (PA + 16 * NTP + 4); }
template <int NTP>
constexpr size_t mask_smem() {
  return size_t(STAGES) * stage_doubles<NTP>() * 8 + 2 * STAGES * 8 + STAGES * 8;
}

struct MaskArgs {
  double* c;
  size_t ldc;
  const double* at;  // [k][pitch_a], rows 16-byte aligned
  size_t pitch_a;
  int acols;         // columns of a row that may be copied (>= m, even)
  const double* b;   // [k][pitch_b], pieces 16-byte aligned
  size_t pitch_b;
  int blk_pitch;     // columns from one block to the next in b
  int bcols;         // columns of a row that may be copied (even)
  const double* zero;  // TM zeros: the row past a list's end
  const int* lists;    // [nblk][k]
  const int* counts;
  int m, n, k, blk, nblk, nsub, sw, tiles_m;
  int cvec;            // C rows take 16-byte accesses at every piece
  int* counter;
  const int* compact;  // 0: the dense form runs instead
};

__device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity, int code) {
  return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, &g_mask_error, code));
}

// NTP: pairs of n8 tiles per item, i.e. 16 * NTP columns.  kLate: the next item is drawn
// after this one's copies instead of before them (see draws_late; a template argument,
// because a branch on it in the kernel cost 3 % of every product).
template <int NTP, bool kLate>
__global__ void __launch_bounds__(THREADS, 2)
dgemm_mask_kernel(const __grid_constant__ MaskArgs p) {
  constexpr int PB = 16 * NTP + 4;
  constexpr int SD = stage_doubles<NTP>();
  extern __shared__ __align__(128) double mask_smem_raw[];
  double* sm = mask_smem_raw;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + STAGES * SD);
  uint64_t* empty = full + STAGES;
  int2* info = reinterpret_cast<int2*>(empty + STAGES);  // (item or -1, rows | last << 8)

  if (*p.compact == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], CONS);
    }
    tc::mbar_fence_init();
  }
  __syncthreads();
  const int total = p.nblk * p.nsub * p.tiles_m;

  if (warp == CONS) {
    // ------------------------------- producer -------------------------------
    int fill = 0;
    bool ok = true;
    int it = 0;
    if (lane == 0) it = atomicAdd(p.counter, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    while (ok && it < total) {
      int next = 0;
      if (!kLate && lane == 0) next = atomicAdd(p.counter, 1);
      const int mt = it % p.tiles_m, piece = it / p.tiles_m;
      const int b = piece / p.nsub, sub = piece % p.nsub;
      const int nb = p.counts[b];
      const int off = sub * p.sw;
      const int x0 = b * p.blk_pitch + off;
      const int w = min(min(p.sw, p.blk_pitch - off), p.bcols - x0);
      const int m0 = mt * TM;
      const uint32_t ab = uint32_t(min(TM, p.acols - m0)) * 8, bb = uint32_t(w) * 8;
      const int* I = p.lists + size_t(b) * p.k;
      const int r = lane & 15;
      const int nch = w > 0 ? (nb + TK - 1) / TK : 0;
      int v = r < nb ? I[r] : -1;
      for (int kc = 0; kc < nch; ++kc, ++fill) {
        const int row = v;
        const int kn = (kc + 1) * TK + r;
        v = kn < nb ? I[kn] : -1;
        const int s = fill % STAGES;
        if (fill >= STAGES && !wait_all(&empty[s], ((fill / STAGES) - 1) & 1, 0x5101)) {
          ok = false;
          break;
        }
        double* st = sm + s * SD;
        if (lane == 0) {
          info[s] = make_int2(it, min(TK, nb - kc * TK) | (kc + 1 == nch ? 256 : 0));
          tc::mbar_arrive_expect_tx(&full[s], TK * (ab + bb));
        }
        __syncwarp();
        if (lane < TK)
          tc::bulk_load(st + r * PA, row >= 0 ? p.at + size_t(row) * p.pitch_a + m0 : p.zero, ab,
                        &full[s]);
        else
          tc::bulk_load(st + TK * PA + r * PB,
                        row >= 0 ? p.b + size_t(row) * p.pitch_b + x0 : p.zero, bb, &full[s]);
      }
      if (kLate && lane == 0) next = atomicAdd(p.counter, 1);
      it = __shfl_sync(0xffffffffu, next, 0);
    }
    if (ok) {  // the end mark
      const int s = fill % STAGES;
      if (fill < STAGES || wait_all(&empty[s], ((fill / STAGES) - 1) & 1, 0x5101)) {
        if (lane == 0) {
          info[s] = make_int2(-1, 0);
          tc::mbar_arrive(&full[s]);
        }
        ++fill;
      }
    }
    // every copy lands before the CTA exits
    if (lane == 0)
      for (int f = max(0, fill - STAGES); f < fill; ++f)
        tc::mbar_wait(&full[f % STAGES], (f / STAGES) & 1, &g_mask_error, 0x5103, true);
    return;
  }

  // ------------------------------- consumers -------------------------------
  const int g = lane >> 2, q = lane & 3;
  const int ra = warp * 16 + 2 * g;
  double acc[2 * NTP][4];
#pragma unroll
  for (int j = 0; j < 2 * NTP; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;

  for (int use = 0;; ++use) {
    const int s = use % STAGES;
    if (!wait_all(&full[s], (use / STAGES) & 1, 0x5102)) break;
    const int2 in = info[s];
    if (in.x < 0) break;
    const double* As = sm + s * SD;
    const double* Bs = As + TK * PA;
    const int kend = (in.y & 255) > 8 ? TK : 8;
#pragma unroll
    for (int kk = 0; kk < TK; kk += 8) {
      if (kk >= kend) break;
      const double2 lo = *reinterpret_cast<const double2*>(As + (kk + q) * PA + ra);
      const double2 hi = *reinterpret_cast<const double2*>(As + (kk + q + 4) * PA + ra);
#pragma unroll
      for (int j = 0; j < NTP; ++j) {
        const double2 b0 = *reinterpret_cast<const double2*>(Bs + (kk + q) * PB + 16 * j + 2 * g);
        const double2 b1 =
            *reinterpret_cast<const double2*>(Bs + (kk + q + 4) * PB + 16 * j + 2 * g);
        dmma_16x8x8(acc[2 * j], lo.x, lo.y, hi.x, hi.y, b0.x, b1.x);
        dmma_16x8x8(acc[2 * j + 1], lo.x, lo.y, hi.x, hi.y, b0.y, b1.y);
      }
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&empty[s]);
    if (!(in.y & 256)) continue;

    // C += the item's products.  Row g (g + 8) of the m16 tile is row 2g (2g + 1)
    // of the 16, column x of n8 tile 2j + e is column 2x + e of the 16.
    const int mt0 = in.x % p.tiles_m, piece = in.x / p.tiles_m;
    const int b = piece / p.nsub, sub = piece % p.nsub;
    const int col0 = b * p.blk + sub * p.sw;
    const int wc = min(min(p.sw, p.blk - sub * p.sw), p.n - col0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = mt0 * TM + ra + h;
      if (row >= p.m) continue;
      double* crow = p.c + size_t(row) * p.ldc + col0 + 4 * q;
      if (p.cvec) {
        double2 old[NTP][2];
#pragma unroll
        for (int j = 0; j < NTP; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)  // wc is even where cvec is set
            if (16 * j + 4 * q + 2 * e < wc)
              old[j][e] = *reinterpret_cast<const double2*>(crow + 16 * j + 2 * e);
#pragma unroll
        for (int j = 0; j < NTP; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (16 * j + 4 * q + 2 * e < wc)
              *reinterpret_cast<double2*>(crow + 16 * j + 2 * e) = make_double2(
                  old[j][e].x + acc[2 * j][2 * h + e], old[j][e].y + acc[2 * j + 1][2 * h + e]);
      } else {
#pragma unroll
        for (int j = 0; j < NTP; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (16 * j + 4 * q + e < wc) crow[16 * j + e] += acc[2 * j + (e & 1)][2 * h + (e >> 1)];
      }
    }
#pragma unroll
    for (int j = 0; j < 2 * NTP; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;
  }
}

// Chooses between the compacted and the dense form by the share of present
// tiles (max_share >= 1: always compacted), resets the item counter, clears the
// zero row.
__global__ void __launch_bounds__(256)
mask_setup(const int* __restrict__ counts, int nblk, int k, double max_share, int* counter,
           int* compact, double* zero) {
  __shared__ unsigned long long sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  unsigned long long mine = 0;
  for (int b = threadIdx.x; b < nblk; b += 256) mine += counts[b];
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, mine);
  for (int i = threadIdx.x; i < TM; i += 256) zero[i] = 0.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    *counter = 0;
    *compact = max_share >= 1.0 || double(sum) <= max_share * double(nblk) * double(k) ? 1 : 0;
  }
}

// The present tiles of B into rows of nblk * blk_pitch columns (blk_pitch = blk
// rounded up to even): dst[p][b * blk_pitch + j] = src[p*ld + b*blk + j].  Four rows at a
// time (one: 100 x 16384 x 3000, odd rows, 0.3 present 430 us the call, now 257).
__global__ void __launch_bounds__(256)
pack_tiles(double* __restrict__ dst, const double* __restrict__ src, size_t ld, int n, int k,
           int blk, int blk_pitch, int nblk, const uint8_t* __restrict__ tab, size_t ldtab,
           const int* __restrict__ compact) {
  if (*compact == 0) return;
  const long long cols = (long long)nblk * blk_pitch;
  const long long x = (long long)blockIdx.x * 256 + threadIdx.x;
  if (x >= cols) return;
  const int b = int(x / blk_pitch), j = int(x % blk_pitch);
  const int col = b * blk + j;
  const bool in = j < blk && col < n;
  for (int p0 = blockIdx.y; p0 < k; p0 += 4 * gridDim.y) {
    bool on[4];
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = p0 + i * gridDim.y;
      on[i] = p < k && tab[size_t(p) * ldtab + b];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = on[i] && in ? src[size_t(p0 + i * gridDim.y) * ld + col] : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (on[i]) dst[size_t(p0 + i * gridDim.y) * cols + x] = v[i];
  }
}

int sm_count() {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nsm;
}

// Whether the items are so few that up to half of the CTAs get a second one.  Drawn before
// the first one's copies, the rest went to the CTAs that start first, or both to one SM,
// while others had none.  16384 columns x 2228, us, drawn before / after the copies: 8 rows
// (1.2 items to a CTA), 0.3 present 186 / 136, all 550 / 383; 60 rows, 4000 columns (0.3)
// 160 / 116; but 300 rows (3.5), 0.6 565 / 610, 500 rows, 8000 columns (1.7) 156 / 170.
bool draws_late(long long items, int ctas) { return items <= ctas + ctas / 2; }

template <int NTP, bool kLate>
cudaError_t launch_form(const MaskArgs& a, int ctas, cudaStream_t stream) {
  constexpr size_t smem = mask_smem<NTP>();
  static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs per SM");
  cudaError_t err = cudaFuncSetAttribute(dgemm_mask_kernel<NTP, kLate>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (err != cudaSuccess) return err;
  dgemm_mask_kernel<NTP, kLate><<<ctas, THREADS, smem, stream>>>(a);
  return cudaGetLastError();
}

template <int NTP>
cudaError_t launch_mask(const MaskArgs& a, cudaStream_t stream) {
  const int nsm = sm_count();
  if (nsm <= 0) return cudaErrorInvalidDevice;
  const long long total = (long long)a.nblk * a.nsub * a.tiles_m;
  const int ctas = int(std::min<long long>(total, 2 * nsm));
  return draws_late(total, ctas) ? launch_form<NTP, true>(a, ctas, stream)
                                 : launch_form<NTP, false>(a, ctas, stream);
}

size_t a256(size_t x) { return (x + 255) / 256 * 256; }

bool al16(const void* p, size_t ld) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 2 == 0;
}

// Columns a CTA forms for a piece of `width` columns in `nsub` equal pieces.
int padded(int width, int nsub) { return nsub * (((width + nsub - 1) / nsub + 15) / 16 * 16); }

// The pieces of up to MAXW columns that a block of `width` columns is cut into:
// the count, from the least possible to two more, that pads the least (240
// columns: five of 48, not four of 60 padded to 64).
int pieces(int width) {
  const int least = (width + MAXW - 1) / MAXW;
  int best = least;
  for (int x = least + 1; x <= least + 2; ++x)
    if (padded(width, x) < padded(width, best)) best = x;
  return best;
}

// Where A^T and B come from, the pieces of a column block, and the scratch.
struct MaskPlan {
  bool a_inplace, b_inplace;
  int nblk, nsub, sw, blk_pitch;
  size_t pitch_a, at, bp, lists, counts, counter, zero, total;
};

MaskPlan mask_plan(const double* a, const double* b, int m, int n, int k, size_t lda, size_t ldb,
                   bool transa, int blk) {
  MaskPlan P{};
  P.a_inplace = transa && al16(a, lda) && m % 2 == 0;
  P.b_inplace = al16(b, ldb) && blk % 2 == 0 && n % 2 == 0;
  P.nblk = int(((long long)n + blk - 1) / blk);
  const int width = std::min(blk, n);  // a block wider than C has only n columns
  P.nsub = pieces(width);
  P.sw = ((width + P.nsub - 1) / P.nsub + 1) / 2 * 2;
  P.blk_pitch = P.b_inplace ? blk : (std::min(blk, n) + 1) / 2 * 2;
  P.pitch_a = P.a_inplace ? lda : size_t((m + 15) / 16 * 16);
  P.at = 0;
  P.bp = P.at + (P.a_inplace ? 0 : a256(size_t(k) * P.pitch_a * 8));
  P.lists = P.bp + (P.b_inplace ? 0 : a256(size_t(k) * P.nblk * P.blk_pitch * 8));
  P.counts = P.lists + a256(size_t(P.nblk) * k * sizeof(int));
  P.counter = P.counts + a256(size_t(P.nblk) * sizeof(int));
  P.zero = P.counter + 256;
  P.total = P.zero + a256(TM * sizeof(double));
  return P;
}

}  // namespace

bool dgemm_mask_applies(int m, int n, int k, int blk) {
  const long long width = std::min(blk, n), nsub = pieces(int(width));
  const long long nblk = ((long long)n + blk - 1) / blk;
  const long long items = nblk * nsub * ((m + TM - 1) / TM);
  // narrow blocks fill too little of a tile
  if (width < 32) return false;
  // up to here the dense form over zero-filled tiles is over before the lists are
  // made and their items run: 200 x 1000 x 200 takes 18 us against 24 to 34 here
  // (15 % to all tiles present), 300 x 2000 x 300 36 against 25 to 43,
  // 600 x 1500 x 600 68 against 39 to 107, 500 x 8000 x 500 174 against 56 to 164
  if (2.0 * m * n * k <= 4e8) return false;
  // index and grid limits
  return items < (1ll << 30) && nblk < (1 << 24) &&
         nblk * (blk + 1ll) < (1ll << 31) && k <= 500000 && m <= 2000000;
}

// What the compacted form takes, for the choice between it and the dense one.  An SM's CTAs
// form 34 TFLOP/s of padded products between them (a piece's columns by 16, rows of C by
// 128), and the SM with the most items decides: one item alone takes 1.25 times an item's
// share of a pair of CTAs, two take two.  Before that come the lists with their launches, and
// the copies of operands that are not used in place.  us in the dense form / this one at 0.5
// present / at 1.0: 2228 x 2000 x 2228, BLKSIZE 48 683 / 442 / 825; 130 x 8000 x 2228 294 /
// 209 / 386; 70 x 16384 x 2228 404 / 213 / 385.  On 22 shapes (m 30 to 5000, n 100 to 16384, k
// 200 to 3000) with 3 to 8 block sizes the model gives 0.90 to 1.02 of what eight in ten of
// them take, 0.70 to 1.13 of all (the least with fewer items than SMs at BLKSIZE 32).
MaskTimes dgemm_mask_times(const double* a, const double* b, int m, int n, int k, size_t lda,
                           size_t ldb, bool transa, int blk) {
  const MaskPlan P = mask_plan(a, b, m, n, k, lda, ldb, transa, blk);
  const int nsm = std::max(sm_count(), 1);
  const long long items = (long long)P.nblk * P.nsub * ((m + TM - 1) / TM);
  const double item = 2.0 * TM * ((P.sw + 15) / 16 * 16) * k / (34e6 / nsm);
  MaskTimes t;
  t.lists = 28.0;
  t.copies = (P.a_inplace ? 0.0 : 16.0 * m * k / 6e6) + (P.b_inplace ? 0.0 : 16.0 * n * k / 3.2e6);
  t.products = item * (items <= nsm ? 1.25 : double((items + nsm - 1) / nsm));
  return t;
}

size_t dgemm_mask_workspace(const double* a, const double* b, int m, int n, int k, size_t lda,
                            size_t ldb, bool transa, int blk) {
  return mask_plan(a, b, m, n, k, lda, ldb, transa, blk).total;
}

cudaError_t dgemm_mask_compact(double* c, const double* a, const double* b, int m, int n, int k,
                               size_t lda, size_t ldb, size_t ldc, bool transa,
                               const uint8_t* tab, size_t ldtab, int blk, double max_share,
                               int* compact, void* workspace, cudaStream_t stream) {
  const MaskPlan P = mask_plan(a, b, m, n, k, lda, ldb, transa, blk);
  char* ws = static_cast<char*>(workspace);
  int* lists = reinterpret_cast<int*>(ws + P.lists);
  int* counts = reinterpret_cast<int*>(ws + P.counts);
  int* counter = reinterpret_cast<int*>(ws + P.counter);
  double* zero = reinterpret_cast<double*>(ws + P.zero);
  cudaError_t err = aodm_block_lists_launch(tab, ldtab, k, P.nblk, lists, counts, stream);
  if (err != cudaSuccess) return err;
  mask_setup<<<1, 256, 0, stream>>>(counts, P.nblk, k, max_share, counter, compact, zero);
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  MaskArgs g{};
  g.c = c;
  g.ldc = ldc;
  g.at = a;
  g.pitch_a = P.pitch_a;
  g.acols = m;
  if (!P.a_inplace) {
    double* at = reinterpret_cast<double*>(ws + P.at);
    if ((err = dgemm_pack_kmajor(at, a, lda, m, k, int(P.pitch_a), transa, compact, stream)) !=
        cudaSuccess)
      return err;
    g.at = at;
    g.acols = int(P.pitch_a);
  }
  g.b = b;
  g.pitch_b = ldb;
  g.bcols = n;
  if (!P.b_inplace) {
    double* bp = reinterpret_cast<double*>(ws + P.bp);
    const long long cols = (long long)P.nblk * P.blk_pitch;
    // a few CTAs per SM's place: those of a form that does not run are soon over
    const long long across = (cols + 255) / 256;
    const unsigned down = unsigned(std::min<long long>((k + 3) / 4, 2048 / across + 1));
    pack_tiles<<<dim3(unsigned(across), down), 256, 0, stream>>>(bp, b, ldb, n, k, blk, P.blk_pitch, P.nblk, tab, ldtab, compact);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    g.b = bp;
    g.pitch_b = size_t(cols);
    g.bcols = int(cols);
  }
  g.blk_pitch = P.blk_pitch;
  g.zero = zero;
  g.lists = lists;
  g.counts = counts;
  g.m = m;
  g.n = n;
  g.k = k;
  g.blk = blk;
  g.nblk = P.nblk;
  g.nsub = P.nsub;
  g.sw = P.sw;
  g.tiles_m = (m + TM - 1) / TM;
  g.cvec = al16(c, ldc) && blk % 2 == 0 && n % 2 == 0;
  g.counter = counter;
  g.compact = compact;
  switch ((P.sw + 15) / 16) {  // a piece of a block of 32 columns or more has over 16
    case 2: return launch_mask<2>(g, stream);
    case 3: return launch_mask<3>(g, stream);
    default: return launch_mask<4>(g, stream);
  }
}

cudaError_t dgemm_mask_reset_error(cudaStream_t stream) {
  static const int zero = 0;
  return cudaMemcpyToSymbolAsync(g_mask_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice,
                                 stream);
}

cudaError_t dgemm_mask_read_error(int* code) {
  return cudaMemcpyFromSymbol(code, g_mask_error, sizeof(int));
}

}  // namespace cfgmm
