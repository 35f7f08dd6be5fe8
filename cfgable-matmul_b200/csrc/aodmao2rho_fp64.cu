// aodmao2rho_fp64.cu -- masked AO-DM-AO contraction in FP64 on the FP64 tensor cores.
//
//   rho[s][g] += sum_{u in I(b)} ao_lhs[u][g] * sum_{v in I(b)} D_s[u][v] * ao_rhs[v][g],
//   b = g / BLK,  I(b) = { u < nao : tab[u*ldtab + b] != 0 } in ascending order.
//
// Semantics follow MatmulLoops::aodmao2rho_loop_parallel
// (src/impl_aodmao2rho.rs:171-244): the per-block active lists are exactly the
// reference's compaction (get_indices_from_non0tab, impl_matmul_non0tab.rs:
// 118-129, applied per block in impl_aodmao2rho.rs:126-133), a block with an
// empty list is skipped, masked (AO, block) entries never contribute whatever
// ao_lhs / ao_rhs hold there, and rho is accumulated into.
//
// Design:
//   1. aodm_block_lists: one CTA per grid block builds I(b) on the device
//      (ballot + popc prefix sums); no host round trip.
//   2. aodm_build_items: one CTA turns the per-block counts into a compact
//      work list (block b, 64-point grid tile, 64-row tile of I(b)) and resets
//      the work counters.
//   3. aodm_fp64_kernel: a persistent kernel, one CTA per SM and group of up
//      to 3 density matrices, that draws work items from the list.  It forms
//      X = D_s[I,I] * ao_rhs[I, tile] on the FP64 tensor cores (DMMA
//      m16n8k4) with the gather done by 8-byte cp.async straight from the
//      compacted index list -- no packed copy of D ever reaches HBM -- and
//      then reduces phi_lhs (.) X over the 64 rows in registers, warp
//      shuffles and shared memory, so X never leaves the SM.  The ao_rhs
//      tile is shared by all density matrices of the group.
//      The active list of the current block is staged in shared memory, so
//      the gather addresses never wait on global loads.
//   3b. aodm_fp64_pipe_kernel: the same items with producer warps (D by
//      cp.async; ao_rhs rows by one bulk copy each where the rows are 16-byte
//      aligned and BLKSIZE is even, by cp.async otherwise) and consumer warps
//      (DMMA m16n8k8) meeting on mbarriers; with a symmetric-D mode.  The
//      form used; form 3 remains for CFGMM_AODM_PIPE=0.
//   4. aodm_reduce: adds the per-row-tile partial sums of each grid tile in a
//      fixed order, so results are deterministic run to run (unlike the
//      reference, whose lock order varies).  In a small single call the warp that
//      stores a grid tile's last partial sums does it (3b).
//   A single call is three launches, or four with 4: lists and symmetry check, work
//   list, 3b.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "aodmao2rho_fp64.cuh"
#include "tcgen05.cuh"

namespace cfgmm {

// Error word of the pipelined kernel's bounded waits (0 = none).
__device__ int g_aodm_error;

namespace {

constexpr int TU = 64;   // compacted rows (u) per work item
constexpr int TG = 64;   // grid points per work item
constexpr int STAGES = 3;
constexpr int THREADS = 256;
constexpr int LIST_CAP = 8192;  // active-list entries staged in shared memory

// ---------------------------------------------------------------------------
// 1. active lists: lists[b*nao + i] = i-th active AO of block b, counts[b]
//    Each of the CTA's eight warps takes an eighth of up to 16384 AOs: the mask
//    bytes are requested eight at a time, their ballots kept in shared memory, and
//    after one barrier each warp writes its part of the list behind the others'.
//    (256 AOs at a time, each with its own loads and three barriers, took 11 us for
//    2228 AOs.)
// ---------------------------------------------------------------------------
constexpr int LIST_WORDS = 64;  // ballots per warp and pass

__device__ __forceinline__ void
block_list(const uint8_t* __restrict__ tab, size_t ldtab, int nao, int b, int* __restrict__ lists,
           int* __restrict__ counts) {
  __shared__ uint32_t words[8][LIST_WORDS];
  __shared__ int warp_tot[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* col = tab + b;
  int* out = lists + size_t(b) * nao;
  int base = 0;
  for (int first = 0; first < nao; first += 8 * 32 * LIST_WORDS) {
    const int left = min(nao - first, 8 * 32 * LIST_WORDS);
    const int nw = (left + 255) / 256;  // ballots of a warp
    const int u0 = first + warp * nw * 32;
    int n = 0;
    for (int i = 0; i < nw; i += 8) {
      uint8_t on[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int u = u0 + (i + q) * 32 + lane;
        on[q] = i + q < nw && u < nao ? col[size_t(u) * ldtab] : 0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t bal = __ballot_sync(0xffffffffu, on[q] != 0);
        n += __popc(bal);
        if (lane == 0 && i + q < nw) words[warp][i + q] = bal;
      }
    }
    if (lane == 0) warp_tot[warp] = n;
    __syncthreads();
    int at = base;
    for (int w = 0; w < 8; ++w) {
      base += warp_tot[w];
      if (w < warp) at += warp_tot[w];
    }
    for (int i = 0; i < nw; ++i) {
      const uint32_t bal = words[warp][i];
      if (bal >> lane & 1u) out[at + __popc(bal & ((1u << lane) - 1u))] = u0 + i * 32 + lane;
      at += __popc(bal);
    }
    __syncthreads();
  }
  if (tid == 0) counts[b] = base;
}

__global__ void __launch_bounds__(256)
aodm_block_lists(const uint8_t* __restrict__ tab, size_t ldtab, int nao, int nblk,
                 int* __restrict__ lists, int* __restrict__ counts) {
  if (int(blockIdx.x) < nblk) block_list(tab, ldtab, nao, blockIdx.x, lists, counts);
}

// Whether tile (by, bx) of d (32 x 32, by <= bx) differs from the transpose of tile
// (bx, by); to every thread of the CTA (256).
__device__ __forceinline__ bool asym_tile(const double* __restrict__ d, size_t stride_ao, int nao,
                                          int bx, int by) {
  __shared__ double tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  // both tiles are requested before the barrier: tile (by, bx) into shared
  // memory, this thread's elements of tile (bx, by) into registers
  double mine[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = ty + 8 * k;
    const int r = by * 32 + i, c = bx * 32 + tx;
    tile[i][tx] = (r < nao && c < nao) ? d[size_t(r) * stride_ao + c] : 0.0;
    const int r2 = bx * 32 + i, c2 = by * 32 + tx;
    mine[k] = (r2 < nao && c2 < nao) ? d[size_t(r2) * stride_ao + c2] : 0.0;
  }
  __syncthreads();
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = ty + 8 * k;
    const int r2 = bx * 32 + i, c2 = by * 32 + tx;
    if (r2 < nao && c2 < nao) bad |= !(mine[k] == tile[tx][i]);
  }
  return __syncthreads_or(bad) != 0;
}

// A single call's first launch: the block lists (CTAs 0 .. nblk-1) and, beside
// them, the symmetry check of every D_s (the `ncheck` CTAs after them, each with
// every ncheck-th of the tile pairs of one s after the other; bad[i] = whether CTA i
// found one that differs).
__global__ void __launch_bounds__(256)
aodm_lists_and_check(const uint8_t* __restrict__ tab, size_t ldtab, int nao, int nblk,
                     int* __restrict__ lists, int* __restrict__ counts,
                     const double* __restrict__ dms, size_t stride_ao, int nset, int ncheck,
                     uint8_t* __restrict__ bad) {
  if (int(blockIdx.x) < nblk) {
    block_list(tab, ldtab, nao, blockIdx.x, lists, counts);
    return;
  }
  const int me = int(blockIdx.x) - nblk;
  const unsigned nt = unsigned(nao + 31) / 32;
  const unsigned pairs = nt * (nt + 1) / 2;  // below 2^32 / nset: D would not fit otherwise
  bool any = false;
  for (unsigned t = me; t < pairs * nset && !any; t += ncheck) {
    const unsigned s = t / pairs, k = t % pairs;  // pair (by <= bx) at bx (bx + 1) / 2 + by
    unsigned bx = unsigned((sqrtf(8.0f * float(k) + 1.0f) - 1.0f) * 0.5f);
    while (bx * (bx + 1) / 2 > k) --bx;
    while ((bx + 1) * (bx + 2) / 2 <= k) ++bx;
    any = asym_tile(dms + size_t(s) * stride_ao * stride_ao, stride_ao, nao, int(bx),
                    int(k - bx * (bx + 1) / 2));
  }
  if (threadIdx.x == 0) bad[me] = any;
}

// ---------------------------------------------------------------------------
// 2. work list: items[i] = (0, b * gsub + gt, utile) for every row tile of every
//    non-empty (block, grid tile); counters[g] = 0.  The items come in order of
//    the row tiles from theirs to the list's end, most first (within one number
//    in no fixed order): in the symmetric mode an item's work is proportional
//    to that number, so the last items drawn are the shortest and the SMs end
//    together.  In block order a taxol-size call's SMs were busy 93 % of the
//    kernel's time, the longest items (129 k cycles) starting at any point.
//    Every item has its own partial-sum slot, so the order changes no result.
//    With `bad` (aodm_lists_and_check's findings) the asymmetry flag is set too.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
aodm_build_items(const int* __restrict__ counts, int nblk, int gsub, int4* __restrict__ items,
                 int* __restrict__ counters, int ncounters, const uint8_t* __restrict__ bad,
                 int ncheck) {
  constexpr int RANKS = 1024;           // longer lists share the first rank
  __shared__ int start[RANKS + 1];      // by tiles left: blocks, then the next free item
  __shared__ int warp_tot[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) g_aodm_error = 0;
  // [ncounters] = total, [ncounters + 1] = asymmetry flag
  for (int i = tid; i <= ncounters; i += 1024) counters[i] = 0;
  for (int r = tid; r <= RANKS; r += 1024) start[r] = 0;
  int differs = 0;
  for (int i = tid; i < ncheck; i += 1024) differs |= bad[i];
  differs = __syncthreads_or(differs);
  if (tid == 0) counters[ncounters + 1] = differs != 0;
  // items with r tiles left: one of every block with at least r of them; rank
  // RANKS takes all above it too
  for (int b = tid; b < nblk; b += 1024) {
    const int nt = (counts[b] + TU - 1) / TU;
    if (nt > 0) atomicAdd(&start[min(nt, RANKS)], 1);
  }
  __syncthreads();
  // thread t: rank RANKS - t, scanned from the highest rank down
  const int rank = RANKS - tid;
  int blocks = start[rank];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, blocks, o);
    if (lane >= o) blocks += v;
  }
  if (lane == 31) warp_tot[warp] = blocks;
  __syncthreads();
  // of the warps before, by lanes (a loop over them took 1 us of the two scans)
  auto before = [&] { return __reduce_add_sync(0xffffffffu, lane < warp ? warp_tot[lane] : 0); };
  blocks += before();  // blocks with >= rank tiles
  int mine = blocks;
  if (tid == 0)  // rank RANKS: every tile from the RANKS-th on
    for (int b = 0; mine && b < nblk; ++b) mine += max(0, (counts[b] + TU - 1) / TU - RANKS);
  int incl = mine;
  __syncthreads();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  incl += before();
  start[rank] = (incl - mine) * gsub;
  if (tid == 1023) counters[ncounters] = incl * gsub;  // rank 1: the total
  __syncthreads();
  for (int b = tid; b < nblk; b += 1024) {
    const int nt = (counts[b] + TU - 1) / TU;
    // .w of entry bg: the main kernel's ticket of block tile bg (its own or another
    // item's entry, zero either way)
    for (int gt = 0; gt < gsub; ++gt) items[b * gsub + gt].w = 0;
    for (int u = 0; u < nt; ++u) {
      const int at = atomicAdd(&start[min(nt - u, RANKS)], gsub);
      for (int gt = 0; gt < gsub; ++gt) items[at + gt] = make_int4(0, b * gsub + gt, u, 0);
    }
  }
}

// ---------------------------------------------------------------------------
// 3. main kernel
// ---------------------------------------------------------------------------
template <int NS, int TKT>
__global__ void __launch_bounds__(THREADS, 1) aodm_fp64_kernel(AodmArgs p) {
  extern __shared__ __align__(128) double smem[];
  constexpr int D_TILE = TU * TKT;  // one D tile per set
  constexpr int P_TILE = TG * TKT;  // ao_rhs tile, stored [g][k]
  constexpr int STAGE = NS * D_TILE + P_TILE;
  constexpr int DC = TKT;           // D gather: threads per row (= columns of a chunk)
  constexpr int DR = THREADS / DC;  // D gather: rows per pass
  constexpr int PR = THREADS / TG;  // ao_rhs gather: k rows per pass
  int* list_s = reinterpret_cast<int*>(smem + STAGES * STAGE);  // LIST_CAP entries
  __shared__ int item_s;
  __shared__ long long key_s;

  const int set0 = blockIdx.y * NS;
  const int total = p.counters[p.ngroups];
  int* counter = p.counters + blockIdx.y;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3;  // 2 x 4 warps; warp tile 32 (u) x 16 (g)
  const int g = lane >> 2, q = lane & 3;
  const int c_d = tid % DC, r_d0 = tid / DC;  // D gather: column c_d, rows r_d0 + DR*i
  const int j_p = tid % TG, c_p0 = tid / TG;  // ao_rhs gather: point j_p, k rows c_p0 + PR*i

  if (tid == 0) key_s = -1;
  for (;;) {
    if (tid == 0) item_s = atomicAdd(counter, 1);
    __syncthreads();  // also orders this item's smem use after the previous one's
    const int it = item_s;
    if (it >= total) break;
    const int4 w = p.items[it];
    const AodmBatch& B = p.batches ? p.batches[w.x] : p.one;
    const int ns = min(NS, B.nset - set0);
    if (ns <= 0) continue;  // this batch has fewer density matrices
    const int bg = w.y, utile = w.z;
    const int b = bg / p.gsub, gt = bg % p.gsub;
    const int nb = B.counts[b];
    const int* Ig = B.lists + size_t(b) * p.nao;
    const bool staged = nb <= LIST_CAP;
    const long long key = (long long)w.x << 32 | b;  // (batch, block) whose list is staged
    if (staged && key_s != key) {
      for (int i = tid; i < nb; i += THREADS) list_s[i] = Ig[i];
      __syncthreads();
      if (tid == 0) key_s = key;
    }
    const int* I = staged ? list_s : Ig;
    const int u0 = utile * TU;
    const int g0 = b * p.blk + gt * TG;
    const int gw = min(min((b + 1) * p.blk, B.ngrid), g0 + TG) - g0;
    const int mu = min(TU, nb - u0);
    const bool jok = j_p < gw;

    int urow[TU / DR];
#pragma unroll
    for (int i = 0; i < TU / DR; ++i) {
      const int r = r_d0 + DR * i;
      urow[i] = (r < mu) ? I[u0 + r] : -1;
    }

    const int kchunks = (nb + TKT - 1) / TKT;
    auto issue = [&](int kc) {
      double* st = smem + (kc % STAGES) * STAGE;
      const int k0 = kc * TKT;
      const int kw = min(TKT, nb - k0);
      const bool cok = c_d < kw;
      const int vcol = cok ? I[k0 + c_d] : 0;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        double* Ds = st + s * D_TILE;
        const bool sok = s < ns;
        const double* dm = p.dms + size_t(set0 + (sok ? s : 0)) * p.dm_stride;
#pragma unroll
        for (int i = 0; i < TU / DR; ++i) {
          const int r = r_d0 + DR * i;
          const bool ok = sok && cok && urow[i] >= 0;
          const double* src = ok ? dm + size_t(urow[i]) * p.stride_ao + vcol : p.dms;
          cp_async_8(Ds + swz<TKT>(r, c_d), src, ok);
        }
      }
      double* Ps = st + NS * D_TILE;
#pragma unroll
      for (int i = 0; i < TKT / PR; ++i) {
        const int c = c_p0 + PR * i;
        const bool ok = jok && c < kw;
        const double* src =
            ok ? B.ao_rhs + size_t(I[k0 + c]) * B.stride_grid + (g0 + j_p) : B.ao_rhs;
        cp_async_8(Ps + swz<TKT>(j_p, c), src, ok);
      }
    };

    double acc[NS][2][2][4];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[s][i][j][e] = 0.0;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
      if (s < kchunks) issue(s);
      cp_async_commit();
    }
    for (int kc = 0; kc < kchunks; ++kc) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      if (kc + STAGES - 1 < kchunks) issue(kc + STAGES - 1);
      cp_async_commit();

      const double* st = smem + (kc % STAGES) * STAGE;
      const double* Ps = st + NS * D_TILE;
#pragma unroll
      for (int kk = 0; kk < TKT; kk += 8) {
        double2 bv[2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
          bv[nt] = *reinterpret_cast<const double2*>(Ps + swz<TKT>(wn * 16 + nt * 8 + g, kk + 2 * q));
        double2 av[NS][2][2];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const double* Ds = st + s * D_TILE;
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const int r = wm * 32 + mt * 16 + g;
            av[s][mt][0] = *reinterpret_cast<const double2*>(Ds + swz<TKT>(r, kk + 2 * q));
            av[s][mt][1] = *reinterpret_cast<const double2*>(Ds + swz<TKT>(r + 8, kk + 2 * q));
          }
        }
        // k-slot .x of every tile of every set, then .y: dependent DMMAs on one
        // accumulator are 4*NS instructions apart.
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
              dmma_16x8x4(acc[s][mt][nt], av[s][mt][0].x, av[s][mt][1].x, bv[nt].x);
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
              dmma_16x8x4(acc[s][mt][nt], av[s][mt][0].y, av[s][mt][1].y, bv[nt].y);
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // stage buffers are reused below

    // Epilogue: rho_part[s][j] = sum_r ao_lhs[I[u0+r]][g0+j] * X[s][r][j].
    // Thread rows: r = wm*32 + mt*16 + g + 8h; columns j = wn*16 + nt*8 + 2q + e.
    double lhs[2][2][2][2];  // [mt][h][nt][e]
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = wm * 32 + mt * 16 + g + 8 * h;
        const bool rok = r < mu;
        const double* row = rok ? B.ao_lhs + size_t(I[u0 + r]) * B.stride_grid : nullptr;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = wn * 16 + nt * 8 + 2 * q + e;
            lhs[mt][h][nt][e] = (rok && j < gw) ? row[g0 + j] : 0.0;
          }
      }
    double* red = smem;  // [NS][2 (wm)][TG]
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double v = 0.0;
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) v = fma(acc[s][mt][nt][2 * h + e], lhs[mt][h][nt][e], v);
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 16);
          if (g == 0) red[(s * 2 + wm) * TG + wn * 16 + nt * 8 + 2 * q + e] = v;
        }
    __syncthreads();
    const size_t slot = B.partial_off + size_t(bg) * p.max_utiles + utile;
    for (int t = tid; t < ns * TG; t += THREADS) {
      const int s = t / TG, j = t % TG;
      p.partial[(slot * p.nset_max + set0 + s) * TG + j] =
          red[(s * 2 + 0) * TG + j] + red[(s * 2 + 1) * TG + j];
    }
    // the __syncthreads at the top of the loop protects `red` and the stages
  }
}

// ---------------------------------------------------------------------------
// 3b. pipelined main kernel: the same work items and partial sums as (3), with
//     the roles split.  Four producer warps gather D_s[I_rows, I(k0..k0+15)]
//     with 8-byte cp.async (lanes along consecutive compacted columns, so a
//     warp's reads coalesce over the runs of active AOs) and sixteen producer
//     lanes fetch the ao_rhs rows I(k0..k0+15) x 64 points, a bulk copy each,
//     into rows of 68 doubles: a quarter warp's 16-byte fragment loads (rows
//     k = q, points 2g and 2g + 1) then meet 8 distinct 16-byte bank groups.
//     (Rows of 64 doubles laid down by TMA gather4 put all four k rows into the
//     same banks: 55 M of the 101 M shared-load wavefronts of a taxol-size call
//     were conflicts.)  Both complete on the stage's mbarrier;
//     eight consumer warps run DMMA m16n8k8 from the stages and release them
//     through a second mbarrier, so the gather of later stages -- and of the
//     next work item -- overlaps the tensor-core work.  The roles meet only on
//     mbarriers, and every wait is bounded (tc::mbar_wait): on a timeout the
//     kernel records a code in g_aodm_error and every warp leaves (exit
//     decisions are made warp-uniform, so no warp-level sync meets an exited
//     lane).
// ---------------------------------------------------------------------------
namespace pipe {
constexpr int TK = 16;         // compacted AOs per stage
constexpr int PSTAGES = 5;     // 6 leaves too little L1 beside shared memory (measured)
constexpr int NPROD = 128;     // producer threads (4 warps)
constexpr int NCONS = 256;     // consumer threads (8 warps, 2 x 4 over rows x points)
constexpr int PTHREADS = NPROD + NCONS;
constexpr int RING = 4;        // work items in flight between the roles
constexpr int D_BYTES = TU * TK * 8;      // one density matrix's tile per stage
constexpr int PHI_PITCH = TG + 4;          // ao_rhs row pitch (doubles), see above
constexpr int PHI_BYTES = TK * PHI_PITCH * 8;
constexpr int RSTEP = NPROD / TK;              // rows apart of one thread's gathers
constexpr int ROWS_PER_THREAD = TU / RSTEP;     // 16

template <int NS>
constexpr int stage_bytes() { return NS * D_BYTES + PHI_BYTES; }

// consumer warp grid: CWM warps along the item's rows x CWN along its points;
// each warp holds MT x NT m16n8 tiles per density matrix.  Four row warps of
// 16 rows share their phi (B) fragments over 32 points: per k step of 8 a warp
// loads 2 A fragment pairs per matrix and 4 B fragment pairs.
constexpr int CWM = 4, CWN = 2;
constexpr int MT = TU / CWM / 16, NT = TG / CWN / 8;

template <int NS>
constexpr int red_doubles() { return 2 * NS * CWM * TG; }  // double-buffered [2][NS][CWM][TG]

template <int NS>
constexpr size_t smem_bytes() {
  return 1024 + size_t(PSTAGES) * stage_bytes<NS>() + size_t(red_doubles<NS>()) * 8 +
         (2 * PSTAGES + 2 * RING + 2) * 8 + RING * 4;
}

// Offset (doubles) of D element (row r, stage column k) in a TU x TK tile.  The
// 16-byte slot c = 4*(k/8) + k%4 holds columns k and k+4 of an 8-column group,
// i.e. the (a0, a2) or (a1, a3) pair of one m16n8k8 A fragment, and the slots
// of each 128-byte row are XOR-swizzled by swz_key(r): a fragment load's
// phases of 8 lanes (rows 2p, 2p+1, slots c0..c0+3) meet 8 distinct slots.
__device__ __forceinline__ int d_off(int r, int k) {
  const int slot = ((k >> 3) << 2) | (k & 3);
  return r * TK + ((slot ^ swz_key(r)) << 1) + ((k >> 2) & 1);
}

// wait-site codes recorded in g_aodm_error
enum : int { kErrItemEmpty = 0x4101, kErrItemFull, kErrStageEmpty, kErrStageFull, kErrEpilogue,
             kErrTeardown };

// Decoded work item (both roles decode the same one).
struct Item {
  const AodmBatch* B;
  int ns, bg, utile, nb, u0, mu, g0, gw;
  const int* I;
};

template <int NS>
__device__ __forceinline__ Item decode(const AodmArgs& p, int4 w, int set0) {
  Item t;
  t.B = p.batches ? &p.batches[w.x] : &p.one;
  t.ns = min(NS, t.B->nset - set0);
  t.bg = w.y;
  t.utile = w.z;
  const int b = t.bg / p.gsub, gt = t.bg % p.gsub;
  t.nb = t.B->counts[b];
  t.I = t.B->lists + size_t(b) * p.nao;
  t.u0 = t.utile * TU;
  t.mu = min(TU, t.nb - t.u0);
  t.g0 = b * p.blk + gt * TG;
  t.gw = min(min((b + 1) * p.blk, t.B->ngrid), t.g0 + TG) - t.g0;
  return t;
}

// Point of the tile that accumulator column 2q + e of n8 tile nt holds, in the
// consumer warps' point group wn.
__device__ __forceinline__ int point_of(int wn, int nt, int q, int e) {
  return wn * 8 * NT + (nt >> 1) * 16 + 4 * q + 2 * e + (nt & 1);
}

// Weight of D[u0 + r][u0 + c] in the diagonal tile of the symmetric mode.
__device__ __forceinline__ double sym_factor(int r, int c) {
  return c < r ? 0.0 : (c == r ? 0.5 : 1.0);
}

// rho[j] += sum over u < nt of part[u * step + j], j < width <= 64, by one warp;
// the partial sums come from other SMs (read past L1), eight in flight per lane.
__device__ __forceinline__ void reduce_tile(const double* part, size_t step, int nt, double* rho,
                                            int width, int lane) {
  double v[2] = {0.0, 0.0};
  for (int u = 0; u < nt; u += 4) {
    double x[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        x[i][h] = u + i < nt ? __ldcg(part + size_t(u + i) * step + 32 * h + lane) : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (u + i < nt) v[h] += x[i][h];
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int j = 32 * h + lane;
    if (j < width) rho[j] = v[h] + rho[j];
  }
}

// Bounded wait whose outcome is the same for every lane of the warp.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* err, int code,
                                          uint64_t lim) {
  const bool ok = tc::mbar_wait(bar, parity, err, code, false, lim);
  return __all_sync(0xffffffffu, ok);
}
}  // namespace pipe

template <int NS>
__global__ void __launch_bounds__(pipe::PTHREADS, 1)
aodm_fp64_pipe_kernel(const __grid_constant__ AodmArgs p) {
  using namespace pipe;
  constexpr int SB = stage_bytes<NS>();
  extern __shared__ uint8_t pipe_smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pipe_smem_raw) + 1023) &
                                           ~uintptr_t(1023));
  double* red = reinterpret_cast<double*>(sm + PSTAGES * SB);  // [2][NS][2][TG]
  uint64_t* full = reinterpret_cast<uint64_t*>(red + red_doubles<NS>());
  uint64_t* empty = full + PSTAGES;
  uint64_t* ifull = empty + PSTAGES;
  uint64_t* iempty = ifull + RING;
  uint64_t* epi = iempty + RING;  // [2]
  int* ring = reinterpret_cast<int*>(epi + 2);
  int* err = &g_aodm_error;
  const uint64_t lim = p.wait_ns ? p.wait_ns : tc::kWaitLimitNs;

  const int tid = threadIdx.x, lane = tid & 31;
  const int set0 = blockIdx.y * NS;
  const int total = p.counters[p.ngroups];
  int* counter = p.counters + blockIdx.y;
  const bool sym = p.asym != nullptr && *p.asym == 0;

  if (tid == 0) {
    for (int s = 0; s < PSTAGES; ++s) {
      tc::mbar_init(&full[s], NPROD + 1);     // NPROD cp.async arrivals + the bulk copies' expect_tx
      tc::mbar_init(&empty[s], NCONS / 32);   // one per consumer warp
    }
    for (int r = 0; r < RING; ++r) {
      tc::mbar_init(&ifull[r], 1);
      tc::mbar_init(&iempty[r], PTHREADS / 32);  // every warp reads every item
    }
    for (int e = 0; e < 2; ++e) tc::mbar_init(&epi[e], NCONS);
    tc::mbar_fence_init();
  }
  __syncthreads();

  if (tid < NPROD) {
    // ------------------------------- producers -------------------------------
    const int kcol = tid & (TK - 1);  // stage column gathered by this thread
    const int r0 = tid / TK;          // rows r0 + RSTEP i
    uint32_t fill = 0;                // stage fills issued so far
    for (int n = 0;; ++n) {
      const int slot = n % RING;
      // the next item for every warp of the CTA: the first is the CTA's own, the others
      // are drawn when they are needed (an item drawn ahead waits behind the one
      // being loaded while other CTAs are idle: 38 -> 43 us at 512 AOs x 4096 points)
      if (tid == 0) {
        int it = total;
        if (*reinterpret_cast<volatile int*>(err) == 0 &&
            (n < RING ||
             tc::mbar_wait(&iempty[slot], ((n / RING) - 1) & 1, err, kErrItemEmpty, false, lim)))
          it = min(n == 0 ? int(blockIdx.x) : int(gridDim.x) + atomicAdd(counter, 1), total);
        ring[slot] = it;
        tc::mbar_arrive(&ifull[slot]);
      }
      int it = total;
      if (warp_wait(&ifull[slot], (n / RING) & 1, err, kErrItemFull, lim)) it = ring[slot];
      it = __shfl_sync(0xffffffffu, it, 0);
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&iempty[slot]);
      if (it >= total) break;
      const int4 w = p.items[it];
      const Item t = decode<NS>(p, w, set0);
      // points of the tile that the table holds: none where a wide block's later
      // tiles start past the grid's end; an odd number (the last tile of an odd
      // grid) is no whole number of 16-byte pieces
      const int pts = max(0, min(TG, t.B->ngrid - t.g0));
      const bool bulk = t.B->rhs_bulk && pts % 2 == 0;
      int prow[ROWS_PER_THREAD];  // AO of each gathered row, -1 past the item's rows
#pragma unroll
      for (int i = 0; i < ROWS_PER_THREAD; ++i) {
        const int r = r0 + RSTEP * i;
        prow[i] = r < t.mu ? t.I[t.u0 + r] : -1;
      }
      const int kchunks = (t.nb + TK - 1) / TK;
      const int kc0 = sym ? t.u0 / TK : 0;  // symmetric D: from the tile's own columns on
      // the compacted column index of the next stage is loaded one stage ahead,
      // so the gather addresses never wait for it
      int vnext = t.I[min(kc0 * TK + kcol, t.nb - 1)];
      for (int kc = kc0; kc < kchunks; ++kc, ++fill) {
        const int k = kc * TK + kcol;
        const bool kv = k < t.nb;
        const int v = vnext;  // t.I[min(k, nb - 1)]: the last active AO stands in past the end
        vnext = t.I[min(k + TK, t.nb - 1)];
        const int stage = fill % PSTAGES;
        if (fill >= PSTAGES &&
            !warp_wait(&empty[stage], ((fill / PSTAGES) - 1) & 1, err, kErrStageEmpty, lim)) {
          // nothing is issued for this fill: no asynchronous arrival may be
          // left pending on a barrier that no one waits for when the CTA exits
          break;
        }
        uint8_t* st = sm + stage * SB;
        const double* dm0 = p.dms + size_t(set0) * p.dm_stride + v;
#pragma unroll
        for (int i = 0; i < ROWS_PER_THREAD; ++i) {
          const bool valid = kv && prow[i] >= 0;
          const double* src = valid ? dm0 + size_t(prow[i]) * p.stride_ao : p.dms;
          double* dst = reinterpret_cast<double*>(st) + d_off(r0 + RSTEP * i, kcol);
          // unrolled (a loop over the sets kept one copy's addresses waiting for the
          // last's: 999 -> 975 us at nao 2228, 103 -> 92 at nao 400, 2 sets)
#pragma unroll
          for (int s = 0; s < NS; ++s)
            if (s < t.ns)
              cp_async_8(dst + s * (D_BYTES / 8), src + (valid ? s * p.dm_stride : 0), valid);
        }
        uint8_t* phi = st + NS * D_BYTES;
        if (!bulk) {
          // ao_rhs rows [TK][TG] by cp.async: lanes along points; the row of
          // stage column j comes from lane j of this warp (kcol = lane & 15)
          const int pt = tid & (TG - 1);
          const bool pv = t.g0 + pt < t.B->ngrid;
#pragma unroll
          for (int i = 0; i < TK / (NPROD / TG); ++i) {
            const int j = (tid / TG) + (NPROD / TG) * i;
            const int row = __shfl_sync(0xffffffffu, v, j);
            cp_async_8(reinterpret_cast<double*>(phi) + j * PHI_PITCH + pt,
                       pv ? t.B->ao_rhs + size_t(row) * t.B->stride_grid + t.g0 + pt
                          : t.B->ao_rhs,
                       pv);
          }
        }
        tc::cp_async_arrive_noinc(&full[stage]);
        // test hook: the first stage's last arrival (the bulk copies' expect_tx,
        // or its stand-in) is never made, so the consumers' bounded wait runs out
        const bool withhold = p.inject && fill == 0;
        if (bulk) {
          if (tid < 32 && !withhold) {
            // ao_rhs rows of the stage columns, from the lanes that gather them
            // (lane j < 16 of warp 0 holds column j; D is zero past the list's end)
            if (tid == 0) tc::mbar_arrive_expect_tx(&full[stage], TK * pts * 8);
            __syncwarp();
            if (tid < TK && pts > 0)
              tc::bulk_load(phi + tid * PHI_PITCH * 8,
                            t.B->ao_rhs + size_t(v) * t.B->stride_grid + t.g0, pts * 8,
                            &full[stage]);
          }
        } else if (tid == 0 && !withhold) {
          tc::mbar_arrive(&full[stage]);  // the arrival the expect_tx makes otherwise
        }
      }
    }
    tc::cp_async_wait_all();
    if (tid == 0) {
      // let every bulk copy of the CTA land before the CTA exits
      for (uint32_t f = fill > PSTAGES ? fill - PSTAGES : 0; f < fill; ++f)
        tc::mbar_wait(&full[f % PSTAGES], (f / PSTAGES) & 1, err, kErrTeardown, true, lim);
    }
  } else {
    // ------------------------------- consumers -------------------------------
    const int ct = tid - NPROD;
    const int warp = ct >> 5;
    const int wn = warp % CWN;  // warp tile: rows wm*16*MT.., points wn*8*NT..
    const int g = lane >> 2, q = lane & 3;
    uint32_t use = 0;
    for (int n = 0;; ++n) {
      const int slot = n % RING;
      int it = total;
      if (warp_wait(&ifull[slot], (n / RING) & 1, err, kErrItemFull, lim)) it = ring[slot];
      it = __shfl_sync(0xffffffffu, it, 0);
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&iempty[slot]);
      if (it >= total) break;
      const Item t = decode<NS>(p, p.items[it], set0);
      // the row groups change warps with every item: those with less to do (the
      // diagonal tile's upper rows below, a list's ragged end) are not always on
      // the same schedulers, and the ring of stages lets warps drift apart
      const int wm = (warp / CWN + n) % CWM;

      // the phi_lhs rows of this thread's epilogue (rows wm*16*MT + mt*16 + g + 8h,
      // points point_of(wn, nt, q, e)) are brought into L2 now, so that the
      // epilogue's loads hit while the tensor pipe waits for them
      int urow[MT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = wm * 16 * MT + mt * 16 + g + 8 * h;
          urow[mt][h] = r < t.mu ? t.I[t.u0 + r] : -1;
          if (urow[mt][h] >= 0)
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(
                  t.B->ao_lhs + size_t(urow[mt][h]) * t.B->stride_grid + t.g0 + wn * 8 * NT +
                  nt * 8));
        }

      double acc[NS][MT][NT][4];
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[s][i][j][e] = 0.0;

      const int kchunks = (t.nb + TK - 1) / TK;
      const int kc0 = sym ? t.u0 / TK : 0;
      bool ok = true;
      for (int kc = kc0; kc < kchunks; ++kc, ++use) {
        const int stage = use % PSTAGES;
        if (!warp_wait(&full[stage], (use / PSTAGES) & 1, err, kErrStageFull, lim)) {
          ok = false;
          break;
        }
        const uint8_t* st = sm + stage * SB;
        const double* phi = reinterpret_cast<const double*>(st + NS * D_BYTES);
        // symmetric D, diagonal tile: D' = strict upper triangle + half diagonal;
        // a stage left of all of the warp's rows holds only zeros of it
        const bool diag = sym && kc < kc0 + TU / TK;
        const bool none =
            (diag && (kc - kc0 + 1) * TK <= wm * 16 * MT) || wm * 16 * MT >= t.mu;
        const int kend = none ? 0 : (t.nb - kc * TK > 8 ? TK : 8);
#pragma unroll
        for (int kk = 0; kk < TK; kk += 8) {
          if (kk >= kend) break;
          // tiles 2j and 2j + 1 take the even and the odd points of a group of
          // 16: column x of tile 2j + e is point 2x + e of the group
          double2 b0[NT / 2], b1[NT / 2];
#pragma unroll
          for (int j = 0; j < NT / 2; ++j) {
            const double* at = phi + (kk + q) * PHI_PITCH + wn * 8 * NT + j * 16 + 2 * g;
            b0[j] = *reinterpret_cast<const double2*>(at);
            b1[j] = *reinterpret_cast<const double2*>(at + 4 * PHI_PITCH);
          }
          const int slot8 = ((kk >> 3) << 2) | q;
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const double* Ds = reinterpret_cast<const double*>(st + s * D_BYTES);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              const int r = wm * 16 * MT + mt * 16 + g;
              double2 lo =
                  *reinterpret_cast<const double2*>(Ds + r * TK + ((slot8 ^ swz_key(r)) << 1));
              double2 hi = *reinterpret_cast<const double2*>(
                  Ds + (r + 8) * TK + ((slot8 ^ swz_key(r + 8)) << 1));
              if (diag) {
                const int c = (kc - kc0) * TK + kk + q;  // column within the diagonal tile
                lo.x *= sym_factor(r, c);
                lo.y *= sym_factor(r, c + 4);
                hi.x *= sym_factor(r + 8, c);
                hi.y *= sym_factor(r + 8, c + 4);
              }
#pragma unroll
              for (int j = 0; j < NT / 2; ++j) {
                dmma_16x8x8(acc[s][mt][2 * j], lo.x, hi.x, lo.y, hi.y, b0[j].x, b1[j].x);
                dmma_16x8x8(acc[s][mt][2 * j + 1], lo.x, hi.x, lo.y, hi.y, b0[j].y, b1[j].y);
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[stage]);
      }
      if (!ok) break;

      // rho_part[s][j] = sum_r phi_lhs[I[u0+r]][g0+j] * X[s][r][j]: rows reduced
      // in registers and shuffles, the CWM row groups (wm) through `red`
      double lhs[MT][2][NT][2];  // [mt][h][nt][e]
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double* row =
              urow[mt][h] >= 0 ? t.B->ao_lhs + size_t(urow[mt][h]) * t.B->stride_grid : nullptr;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int j = point_of(wn, nt, q, e);
              lhs[mt][h][nt][e] = (row && j < t.gw) ? row[t.g0 + j] : 0.0;
            }
        }
      double* rb = red + (n & 1) * (NS * CWM * TG);
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            double v = 0.0;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                v = fma(acc[s][mt][nt][2 * h + e], lhs[mt][h][nt][e], v);
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (g == 0) rb[(s * CWM + wm) * TG + point_of(wn, nt, q, e)] = v;
          }
      tc::mbar_arrive(&epi[n & 1]);
      // The buffer is written again two items later, after every consumer has
      // passed the next item's epilogue barrier, i.e. finished reading this one.
      if (!warp_wait(&epi[n & 1], (n >> 1) & 1, err, kErrEpilogue, lim)) break;
      const size_t pslot = t.B->partial_off + size_t(t.bg) * p.max_utiles + t.utile;
      const int nt = (t.nb + TU - 1) / TU;
      // a block tile of one item needs no partial sums (and their fence: 50 AOs x 34863
      // points x 2 67 -> 50 us)
      const bool alone = p.tickets && nt == 1;
      for (int i = ct; i < t.ns * TG; i += NCONS) {
        const int s = i / TG, j = i % TG;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < CWM; ++w) v += rb[(s * CWM + w) * TG + j];
        if (sym) v *= 2.0;
        if (alone) {
          double* r = t.B->rhos + size_t(set0 + s) * t.B->stride_grid + t.g0 + j;
          if (j < t.gw) *r = v + *r;
        } else {
          p.partial[(pslot * p.nset_max + set0 + s) * TG + j] = v;
        }
      }
      if (p.tickets && !alone) {
        // the warp that stores the block tile's last partial sums adds them all into
        // rho, in the fixed order of aodm_reduce
        int ticket = 0;
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          ticket = atomicAdd(&p.tickets[4 * size_t(t.bg)], 1);
        }
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket == nt * (NCONS / 32) * p.ngroups - 1) {
          __threadfence();
          const double* part =
              p.partial + (t.B->partial_off + size_t(t.bg) * p.max_utiles) * p.nset_max * TG;
          for (int s = 0; s < t.B->nset; ++s)
            if (t.gw > 0) reduce_tile(part + s * TG, size_t(p.nset_max) * TG, nt,
                                      t.B->rhos + size_t(s) * t.B->stride_grid + t.g0, t.gw, lane);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// 4. deterministic reduction of the row-tile partials into rho
//    one CTA per (batch, block tile): rpairs[i] = (batch, bg), or bg = i
// ---------------------------------------------------------------------------
__global__ void aodm_reduce(AodmArgs p, const int2* __restrict__ rpairs, int npairs) {
  const int i = blockIdx.x;
  if (i >= npairs) return;
  const int2 pr = rpairs ? rpairs[i] : make_int2(0, i);
  const AodmBatch& B = p.batches ? p.batches[pr.x] : p.one;
  const int bg = pr.y;
  const int b = bg / p.gsub, gt = bg % p.gsub;
  const int nt = (B.counts[b] + TU - 1) / TU;
  if (nt == 0) return;  // fully masked block: rho untouched, as in the reference
  const int g0 = b * p.blk + gt * TG;
  const int gend = min(min((b + 1) * p.blk, B.ngrid), g0 + TG);
  for (int t = threadIdx.x; t < B.nset * TG; t += blockDim.x) {
    const int s = t / TG, j = t % TG;
    if (g0 + j >= gend) continue;
    double v = 0.0;
    for (int u = 0; u < nt; ++u)
      v += p.partial[((B.partial_off + size_t(bg) * p.max_utiles + u) * p.nset_max + s) * TG + j];
    double* r = B.rhos + size_t(s) * B.stride_grid + g0 + j;
    *r = v + *r;
  }
}

__global__ void aodm_reset_counters(int* counters, int ngroups) {
  if (threadIdx.x < ngroups) counters[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    counters[ngroups + 1] = 0;  // asymmetry flag (counters[ngroups] holds the item total)
    g_aodm_error = 0;
  }
}

// *asym = 1 if some D_s differs from its transpose (plans).  Block (bx, by, s)
// with by <= bx compares the 32 x 32 tile (by, bx) with the transpose of (bx, by).
__global__ void __launch_bounds__(256)
aodm_sym_check(const double* __restrict__ dms, size_t stride_ao, size_t dm_stride, int nao,
               int* asym) {
  if (blockIdx.y > blockIdx.x) return;
  if (asym_tile(dms + size_t(blockIdx.z) * dm_stride, stride_ao, nao, blockIdx.x, blockIdx.y) &&
      threadIdx.x == 0)
    atomicOr(asym, 1);
}

template <int NS, int TKT>
cudaError_t launch_main_t(const AodmArgs& a, cudaStream_t stream, bool attrs_only) {
  constexpr size_t smem = size_t(STAGES) * (NS * TU * TKT + TG * TKT) * sizeof(double) +
                          size_t(LIST_CAP) * sizeof(int);
  static_assert(NS * 2 * TG <= STAGES * (NS * TU * TKT + TG * TKT), "reduction buffer fits");
  static_assert(smem <= 227 * 1024, "shared memory budget");
  cudaError_t err = cudaFuncSetAttribute(aodm_fp64_kernel<NS, TKT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (err != cudaSuccess || attrs_only) return err;
  int dev = 0, nsm = 0;
  if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return err;
  aodm_fp64_kernel<NS, TKT><<<dim3(nsm, a.ngroups), THREADS, smem, stream>>>(a);
  return cudaGetLastError();
}

template <int NS>
cudaError_t launch_pipe_t(const AodmArgs& a, cudaStream_t stream, bool attrs_only) {
  constexpr size_t smem = pipe::smem_bytes<NS>();
  static_assert(smem <= 227 * 1024, "shared memory budget");
  cudaError_t err = cudaFuncSetAttribute(aodm_fp64_pipe_kernel<NS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (err != cudaSuccess || attrs_only) return err;
  int dev = 0, nsm = 0;
  if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return err;
  aodm_fp64_pipe_kernel<NS><<<dim3(nsm, a.ngroups), pipe::PTHREADS, smem, stream>>>(a);
  return cudaGetLastError();
}

// The pipelined form is used unless CFGMM_AODM_PIPE=0.
bool pipe_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("CFGMM_AODM_PIPE");
    return !(e && e[0] == '0');
  }();
  return on;
}

}  // namespace

bool aodm_pipe_enabled() { return pipe_enabled(); }

bool aodm_rhs_bulk(const double* ao_rhs, size_t stride_grid, int blk) {
  // every 64-point tile starts at the even point b*blk + 64*gt of a 16-byte
  // aligned row
  return blk % 2 == 0 && reinterpret_cast<uintptr_t>(ao_rhs) % 16 == 0 && stride_grid % 2 == 0;
}

cudaError_t aodm_launch_pipe(const AodmArgs& a, int ns, cudaStream_t stream, bool attrs_only) {
  if (ns == 1) return launch_pipe_t<1>(a, stream, attrs_only);
  if (ns == 2) return launch_pipe_t<2>(a, stream, attrs_only);
  if (ns == 3) return launch_pipe_t<3>(a, stream, attrs_only);
  return cudaErrorInvalidValue;
}

bool aodm_sym_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("CFGMM_AODM_SYM");
    return !(e && e[0] == '0');
  }();
  return on;
}

cudaError_t aodm_launch_sym_check(const double* dms, size_t stride_ao, int nao, int nset,
                                  int* asym, cudaStream_t stream) {
  if (nao <= 0 || nset <= 0) return cudaSuccess;
  const unsigned nt = unsigned((nao + 31) / 32);
  aodm_sym_check<<<dim3(nt, nt, unsigned(nset)), 256, 0, stream>>>(dms, stride_ao,
                                                                  stride_ao * stride_ao, nao, asym);
  return cudaGetLastError();
}

cudaError_t aodm_read_error(int* code) {
  return cudaMemcpyFromSymbol(code, g_aodm_error, sizeof(int));
}

cudaError_t aodm_reset_error(cudaStream_t stream) {
  static const int zero = 0;
  return cudaMemcpyToSymbolAsync(g_aodm_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice,
                                 stream);
}

namespace {
struct WaitInjection {
  bool armed[2] = {false, false};
  unsigned long long ns = 0;
};
thread_local WaitInjection g_wait_injection;
}  // namespace

void arm_wait_injection(int kind, unsigned long long wait_ns) {
  if (kind < 0 || kind > 1) return;
  g_wait_injection.armed[kind] = true;
  g_wait_injection.ns = wait_ns;
}

bool take_wait_injection(int kind, unsigned long long* wait_ns) {
  if (kind < 0 || kind > 1 || !g_wait_injection.armed[kind]) return false;
  g_wait_injection.armed[kind] = false;
  *wait_ns = g_wait_injection.ns;
  return true;
}

int aodm_groups(const AodmConfig& cfg, int nset_max) {
  return (nset_max + cfg.ns - 1) / cfg.ns;
}

AodmConfig aodm_default_config(int nset) {
  return AodmConfig{nset >= 3 ? 3 : nset, 32};
}

cudaError_t aodm_launch_main(const AodmArgs& a, const AodmConfig& cfg, cudaStream_t stream,
                             bool attrs_only) {
  if (cfg.tk == 0) {  // pipelined form
    return aodm_launch_pipe(a, cfg.ns, stream, attrs_only);
  }
  if (cfg.tk == 32) {
    if (cfg.ns == 1) return launch_main_t<1, 32>(a, stream, attrs_only);
    if (cfg.ns == 2) return launch_main_t<2, 32>(a, stream, attrs_only);
    if (cfg.ns == 3) return launch_main_t<3, 32>(a, stream, attrs_only);
  } else if (cfg.tk == 16) {
    if (cfg.ns == 1) return launch_main_t<1, 16>(a, stream, attrs_only);
    if (cfg.ns == 2) return launch_main_t<2, 16>(a, stream, attrs_only);
    if (cfg.ns == 3) return launch_main_t<3, 16>(a, stream, attrs_only);
  }
  return cudaErrorInvalidValue;
}

cudaError_t aodm_launch_reduce(const AodmArgs& a, const int2* rpairs, int npairs,
                               cudaStream_t stream) {
  if (npairs <= 0) return cudaSuccess;
  aodm_reduce<<<npairs, 128, 0, stream>>>(a, rpairs, npairs);
  return cudaGetLastError();
}

cudaError_t aodm_launch_reset(int* counters, int ngroups, cudaStream_t stream) {
  aodm_reset_counters<<<1, 32, 0, stream>>>(counters, ngroups);
  return cudaGetLastError();
}

namespace {
struct Layout {
  size_t lists, counts, items, counters, partial, total;
};

Layout layout(size_t nao, size_t ngrid, size_t nset, size_t blk) {
  const size_t nblk = (ngrid + blk - 1) / blk;
  const size_t gsub = (blk + TG - 1) / TG;
  const size_t max_utiles = (nao + TU - 1) / TU;
  const size_t ngroups = nset;  // upper bound for any set grouping
  auto a256 = [](size_t v) { return (v + 255) / 256 * 256; };
  Layout L;
  L.lists = 0;
  L.counts = L.lists + a256(nblk * nao * sizeof(int));
  L.items = L.counts + a256(nblk * sizeof(int));
  L.counters = L.items + a256(nblk * gsub * max_utiles * sizeof(int4));
  L.partial = L.counters + a256((ngroups + 2) * sizeof(int));  // + item total, asymmetry flag
  L.total = L.partial + nblk * gsub * max_utiles * nset * TG * sizeof(double);
  return L;
}
}  // namespace

cudaError_t aodm_build_items_launch(const int* counts, int nblk, int gsub, int4* items,
                                    int* counters, int ncounters, cudaStream_t stream) {
  aodm_build_items<<<1, 1024, 0, stream>>>(counts, nblk, gsub, items, counters, ncounters,
                                           nullptr, 0);
  return cudaGetLastError();
}

cudaError_t aodm_block_lists_launch(const uint8_t* tab, size_t ldtab, int nao, int nblk,
                                    int* lists, int* counts, cudaStream_t stream) {
  aodm_block_lists<<<nblk, 256, 0, stream>>>(tab, ldtab, nao, nblk, lists, counts);
  return cudaGetLastError();
}

int aodm_row_tile() { return TU; }
int aodm_point_tile() { return TG; }

size_t aodmao2rho_fp64_workspace(size_t nao, size_t ngrid, size_t nset, size_t blk) {
  return layout(nao, ngrid, nset, blk).total;
}

cudaError_t aodmao2rho_fp64(double* rhos, const double* dms, const double* ao_lhs,
                            const double* ao_rhs, size_t stride_ao, size_t stride_grid, int nao,
                            int ngrid, int nset, const uint8_t* tab, size_t ldtab, int blk,
                            void* workspace, cudaStream_t stream) {
  if (nao <= 0 || ngrid <= 0 || nset <= 0) return cudaSuccess;
  const int nblk = (ngrid + blk - 1) / blk;
  const int gsub = (blk + TG - 1) / TG;
  const int max_utiles = (nao + TU - 1) / TU;
  const AodmConfig cfg = aodm_default_config(nset);
  const int ngroups = aodm_groups(cfg, nset);
  const Layout L = layout(nao, ngrid, nset, blk);
  char* ws = static_cast<char*>(workspace);
  int* lists = reinterpret_cast<int*>(ws + L.lists);
  int* counts = reinterpret_cast<int*>(ws + L.counts);
  int4* items = reinterpret_cast<int4*>(ws + L.items);
  int* counters = reinterpret_cast<int*>(ws + L.counters);
  double* partial = reinterpret_cast<double*>(ws + L.partial);

  // the half contraction needs D = D^T and phi_lhs = phi_rhs (one array)
  const bool sym = pipe_enabled() && aodm_sym_enabled() && ao_lhs == ao_rhs;
  // tile pairs to compare, a CTA each up to 16384; their findings wait in the
  // partial sums' place, which is written later
  const long long nt32 = (nao + 31) / 32;
  const int ncheck =
      sym ? int(std::min({nt32 * (nt32 + 1) / 2 * nset, 16384ll, (long long)(L.total - L.partial)}))
          : 0;
  uint8_t* bad = reinterpret_cast<uint8_t*>(partial);
  aodm_lists_and_check<<<unsigned(nblk + ncheck), 256, 0, stream>>>(
      tab, ldtab, nao, nblk, lists, counts, dms, stride_ao, nset, ncheck, bad);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  aodm_build_items<<<1, 1024, 0, stream>>>(counts, nblk, gsub, items, counters, ngroups, bad,
                                           ncheck);
  if ((err = cudaGetLastError()) != cudaSuccess) return err;

  AodmArgs a{};
  a.dms = dms;
  a.stride_ao = stride_ao;
  a.dm_stride = stride_ao * stride_ao;
  a.nao = nao;
  a.blk = blk;
  a.gsub = gsub;
  a.max_utiles = max_utiles;
  a.nset_max = nset;
  a.batches = nullptr;
  a.one = AodmBatch{ao_lhs, ao_rhs, rhos, lists, counts, stride_grid, ngrid, nset, 0};
  a.items = items;
  a.counters = counters;
  a.ngroups = ngroups;
  a.partial = partial;
  if (pipe_enabled()) {
    a.one.rhs_bulk = aodm_rhs_bulk(ao_rhs, stride_grid, blk) ? 1 : 0;
    if (sym) a.asym = counters + ngroups + 1;
    // The kernel's own reduction saves a launch (2 us and the reduction's 5 to 11) and
    // costs each item a fence while its CTA's tensor pipe waits: with at most 4096
    // items (28 per SM) 512 AOs x 4096 points x 1 take 40 us instead of 44; at 8960
    // possible items 2228 AOs x 16384 points x 3 take 1.03 ms with it and 1.01 without.
    if ((long long)nblk * gsub * max_utiles <= 4096) a.tickets = &items[0].w;
    unsigned long long ns = 0;
    if (take_wait_injection(0, &ns)) {  // cfgmm_test_arm_wait_timeout
      a.inject = 1;
      a.wait_ns = ns;
    }
    err = aodm_launch_pipe(a, cfg.ns, stream);
    if (a.tickets) return err;  // rho is reduced
  } else {
    err = aodm_launch_main(a, cfg, stream);
  }
  if (err != cudaSuccess) return err;
  return aodm_launch_reduce(a, nullptr, nblk * gsub, stream);
}

}  // namespace cfgmm
