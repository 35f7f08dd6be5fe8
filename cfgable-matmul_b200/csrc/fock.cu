// fock.cu -- the Fock-build contraction on the per-block compacted AO lists:
//
//   V_s[u][v] += sum_{g in b} phi_lhs[u][g] w_s[g] phi_rhs[v][g],  u, v in I(b),
//
// the transpose of the AO-DM-AO contraction (aodmao2rho_fp64.cu) on its layouts
// and mask: where that one gathers D[I(b), I(b)] as an input, this one scatters
// V[I(b), I(b)] as an output.  Work item = (block, 64-point tile, 64 rows of the
// active list I(b)) for up to 4 weight vectors w_s, the same items as the
// AO-DM-AO kernels (fewer vectors where that would leave a CTA under 8 items to
// draw: 1081 AOs x 3490 points x 4 vectors, 275 items in all, took 189 us with four
// to an item, 167 before vectors were shared).  Only the masked products are formed (a dense product over
// all AO pairs runs ~10x their number on the taxol-size mask).  When phi_lhs and
// phi_rhs are the same array the block's contribution is symmetric in (u, v):
// row tile a then walks the chunks from its own (chunk a) on and adds each
// product of a later chunk to V[u][v] and V[v][u], half the products.  Sums over
// blocks arrive in completion order, so the last bits of V vary from run to run.
//
// One producer warp and eight consumer warps per CTA, two CTAs per SM:
//   * The producer fetches the item's 64 rows of phi_lhs and its weights once,
//     then the compacted columns in chunks of 64 rows of phi_rhs into a ring of
//     two, one bulk copy per row (8-byte cp.async where the rows are not 16-byte
//     aligned).  The columns serve all weight vectors of the item.
//   * Consumer warps (16 rows x 32 columns each) multiply the weights into the
//     phi_lhs fragments, run DMMA m16n8k8 over the tile's points and add the
//     products into V with FP64 atomics (red.add), each warp at its own pace: a
//     warp's atomics overlap the others' DMMAs.
//   * The 16 x 8 fragments are permuted so that a warp's atomics fall into few
//     32-byte sectors: row (column) x of a tile stands for row (column)
//     4 (x % 2) + x / 2 of its 8, and one exchange between lane pairs turns 8
//     rows x 4 columns per instruction into 4 rows x 8 adjacent list columns.
//     A model of the sectors at taxol size: 193 M -> 139 M per call.
//   * Warps whose rows or columns lie past the list's end, and those below the
//     diagonal in the symmetric mode's diagonal tile, skip their products.
// Measured at 2228 AOs x 16384 points x 3 weight vectors (symmetric mode): 1.03 ms;
// 1.52 ms with chunks copied by the computing warps behind CTA barriers, one
// weight vector per item and unpermuted atomics; 1.12 ms before the skips.  What
// bounds it: the FP64 tensor pipe (DMMA; its floor is 0.6 ms), then the L2's atomic
// units (without the atomics the kernel takes 0.15 ms less).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "aodmao2rho_fp64.cuh"
#include "fock.cuh"
#include "tcgen05.cuh"

namespace cfgmm {
namespace {

__device__ int g_fock_error;

constexpr int FT = 64;        // rows per item = columns per chunk = points per tile
constexpr int CONS = 8;       // consumer warps: 4 along rows (16 each) x 2 along columns (32 each)
constexpr int THREADS = 32 * (CONS + 1);
constexpr int NS = kFockVectors;
constexpr int STAGES = 2;     // chunks of phi_rhs in flight
// Row pitch of a staged tile (doubles): 33 16-byte groups, so the 8 lanes of a
// quarter warp's fragment load (rows r and r + 4, point pairs q = 0..3) meet 8
// distinct groups modulo 8.
constexpr int PITCH = FT + 2;
constexpr int TILE = FT * PITCH;
constexpr size_t FOCK_SMEM =
    (size_t(1 + STAGES) * TILE + NS * FT) * 8 + (2 + 2 * STAGES) * 8 + 8 * sizeof(int);

struct FockArgs {
  double* v;
  size_t stride_ao, v_stride;  // v_stride = stride_ao^2
  const double* w;
  const double* ao_lhs;
  const double* ao_rhs;
  size_t stride_grid;
  const int* lists;  // [nblk][nao]
  const int* counts;
  int nao, ngrid, nset, blk, gsub;
  int sym;  // ao_lhs == ao_rhs: chunks from the row tile's own on, mirrored
  int vec;  // phi rows and w 16-byte aligned at every tile
  const int4* items;
  int* counters;  // the work counter (64 bits), the item total
  int ctas;       // that the rule of sharing counts on (the grid may be smaller)
};

__device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity, int code) {
  return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, &g_fock_error, code));
}

// 8-byte asynchronous copy to a shared address, of which the first `bytes` (0 or 8) are
// read; zeros for the rest.
__device__ __forceinline__ void cp_async_8_n(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}

// One item as the producer decodes it for the consumers; bg < 0: no more items.
struct FockItem {
  int bg, nb, u0, gw, b, set0, ns;
};

__global__ void __launch_bounds__(THREADS, 2)
fock_compact_kernel(const __grid_constant__ FockArgs p) {
  extern __shared__ __align__(128) double fock_smem[];
  double* As = fock_smem;                 // [64][PITCH] phi_lhs rows
  double* Bs = As + TILE;                 // [STAGES][64][PITCH] phi_rhs rows
  double* Ws = Bs + STAGES * TILE;        // [NS][64]
  uint64_t* afull = reinterpret_cast<uint64_t*>(Ws + NS * FT);
  uint64_t* aempty = afull + 1;
  uint64_t* full = aempty + 1;            // [STAGES]
  uint64_t* empty = full + STAGES;        // [STAGES]
  FockItem* item = reinterpret_cast<FockItem*>(empty + STAGES);

  // the items once for each group of weight vectors
  const int items = p.counters[2];
  const FockShare share = fock_share(items, p.nset, p.ctas);
  const int per_group = share.per_group;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    // the producer's 32 lanes and one more arrival: the bulk copies' expect_tx
    tc::mbar_init(afull, 33);
    tc::mbar_init(aempty, CONS);
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 33);
      tc::mbar_init(&empty[s], CONS);
    }
    tc::mbar_fence_init();
  }
  __syncthreads();

  if (warp == CONS) {
    // ------------------------------- producer -------------------------------
    auto* counter = reinterpret_cast<unsigned long long*>(p.counters);
    // the first item is the CTA's own, the others are drawn: no round trip to L2 at the
    // start, and the heaviest items one to an SM (1000 AOs, 1000 points, all present 107 ->
    // 93 us; 100 x 5000 21.8 -> 21.2)
    long long it = blockIdx.x;
    int fill = 0, n = 0;
    bool ok = true;
    // rows lane and lane + 32 of `rows` table rows (lane r, r + 32: AOs v0, v1)
    // into a staged tile: `gw` points from g0, none past the rows
    auto rows_in = [&](double* dst, const double* ao, int v0, int v1, int rows, int g0, int gw,
                       uint64_t* bar, bool bulk, uint32_t extra) {
      if (bulk) {
        if (lane == 0) tc::mbar_arrive_expect_tx(bar, uint32_t(rows) * gw * 8 + extra);
        __syncwarp();
        if (lane < rows)
          tc::bulk_load(dst + lane * PITCH, ao + size_t(v0) * p.stride_grid + g0, gw * 8, bar);
        if (lane + 32 < rows)
          tc::bulk_load(dst + (lane + 32) * PITCH, ao + size_t(v1) * p.stride_grid + g0, gw * 8,
                        bar);
      } else {
        // copies past gw read nothing; one warp issues them all, so a row takes as few
        // instructions as it can (193 AOs, 589 points, 2 vectors: 25.2 -> 21.1 us against an
        // address chosen for each copy)
        const double* from = ao + g0 + lane;
        const int lo = lane < gw ? 8 : 0, hi = lane + 32 < gw ? 8 : 0;
        uint32_t to = tc::smem_u32(dst + lane);
#pragma unroll 8
        for (int r = 0; r < rows; ++r, to += PITCH * 8) {
          const int v = __shfl_sync(0xffffffffu, r < 32 ? v0 : v1, r & 31);
          cp_async_8_n(to, from + size_t(v) * p.stride_grid, lo);
          cp_async_8_n(to + 256, from + size_t(v) * p.stride_grid + 32, hi);
        }
        if (lane == 0) tc::mbar_arrive(bar);  // in the expect_tx's place
      }
    };
    while (ok && it < share.total) {
      const int group = it >> 32 ? int(it / items) : int(unsigned(it) / unsigned(items));
      const int4 wi = p.items[it - (long long)group * items];
      const int set0 = group * per_group;
      const int ns = min(per_group, p.nset - set0);
      const int b = wi.y / p.gsub, gt = wi.y % p.gsub, a = wi.z;
      const int nb = p.counts[b];
      const int* I = p.lists + size_t(b) * p.nao;
      const int u0 = a * FT, mu = min(FT, nb - u0);
      const int g0 = b * p.blk + gt * FT;
      const int gw = min(min((b + 1) * p.blk, p.ngrid), g0 + FT) - g0;
      // a wide block's later tiles may start past the grid's end, the last groups past
      // the vectors' (5 in 4 groups of 2)
      if (gw > 0 && ns > 0) {
        const bool bulk = p.vec && gw % 2 == 0;
        const int nch = (nb + FT - 1) / FT, ch0 = p.sym ? a : 0;
        const int ua = I[min(u0 + lane, nb - 1)], ub = I[min(u0 + lane + 32, nb - 1)];
        int va = I[min(ch0 * FT + lane, nb - 1)], vb = I[min(ch0 * FT + lane + 32, nb - 1)];
        for (int ch = ch0; ch < nch && ok; ++ch, ++fill) {
          const int v0 = va, v1 = vb, c1 = (ch + 1) * FT + lane;
          va = I[min(c1, nb - 1)];
          vb = I[min(c1 + 32, nb - 1)];
          const int s = fill % STAGES;
          if (fill >= STAGES && !wait_all(&empty[s], ((fill / STAGES) - 1) & 1, 0x6101)) {
            ok = false;
            break;
          }
          rows_in(Bs + s * TILE, p.ao_rhs, v0, v1, min(FT, nb - ch * FT), g0, gw, &full[s], bulk,
                  0);
          if (bulk)
            tc::mbar_arrive(&full[s]);
          else
            tc::cp_async_arrive_noinc(&full[s]);
          if (ch == ch0) {  // the item's own rows, behind its first chunk
            if (n > 0 && !wait_all(aempty, (n - 1) & 1, 0x6102)) {
              ok = false;
              ++fill;
              break;
            }
            if (lane == 0) *item = FockItem{wi.y, nb, u0, gw, b, set0, ns};
            rows_in(As, p.ao_lhs, ua, ub, mu, g0, gw, afull, bulk, uint32_t(ns) * gw * 8);
            if (bulk) {
              if (lane < ns)
                tc::bulk_load(Ws + lane * FT, p.w + size_t(set0 + lane) * p.stride_grid + g0,
                              gw * 8, afull);
              tc::mbar_arrive(afull);
            } else {
              for (int s2 = 0; s2 < ns; ++s2)
#pragma unroll
                for (int k = lane; k < FT; k += 32)
                  cp_async_8(Ws + s2 * FT + k,
                             k < gw ? p.w + size_t(set0 + s2) * p.stride_grid + g0 + k : p.w,
                             k < gw);
              tc::cp_async_arrive_noinc(afull);
            }
            ++n;
          }
        }
      }
      // the next item only now: its chunks are staged two ahead of the products, which
      // hides the draw, and one drawn earlier would wait behind this one's
      if (lane == 0) it = (long long)(gridDim.x + atomicAdd(counter, 1ull));
      it = __shfl_sync(0xffffffffu, it, 0);
    }
    if (ok && (n == 0 || wait_all(aempty, (n - 1) & 1, 0x6102))) {  // the end mark
      if (lane == 0) {
        item->bg = -1;
        tc::mbar_arrive(afull);
      }
      __syncwarp();
      tc::mbar_arrive(afull);
      ++n;
    }
    // every copy lands before the CTA exits
    tc::cp_async_wait_all();
    if (lane == 0) {
      for (int f = max(0, fill - STAGES); f < fill; ++f)
        tc::mbar_wait(&full[f % STAGES], (f / STAGES) & 1, &g_fock_error, 0x6105, true);
      if (n > 0) tc::mbar_wait(afull, (n - 1) & 1, &g_fock_error, 0x6106, true);
    }
    return;
  }

  // ------------------------------- consumers -------------------------------
  const int wm = warp >> 1;
  const int g = lane >> 2, q = lane & 3;
  const int rg = 4 * (g & 1) + (g >> 1);  // row (column) of its 8 that index g stands for
  const bool odd = g & 1;
  const int r_lo = wm * 16 + rg;
  int use = 0;
  for (int n = 0;; ++n) {
    if (!wait_all(afull, n & 1, 0x6103)) break;
    const FockItem t = *item;
    if (t.bg < 0) break;
    // the columns' halves change sides with every item: the warps that have less
    // to do (a list's ragged end, the diagonal tile) are not always on the same
    // two of the SM's four schedulers
    const int wn = (warp ^ n) & 1;
    const int* I = p.lists + size_t(t.b) * p.nao;
    // this lane's rows (u), and those of its pair of lanes (g even, g odd)
    int u_own[2], u_ev[2], u_od[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = t.u0 + r_lo + 8 * h;
      u_own[h] = r < t.nb ? I[r] : -1;
      u_ev[h] = __shfl_sync(0xffffffffu, u_own[h], lane & ~4);
      u_od[h] = __shfl_sync(0xffffffffu, u_own[h], lane | 4);
    }
    const int ksteps = (t.gw + 7) / 8;
    const int nch = (t.nb + FT - 1) / FT, a = t.u0 / FT, ch0 = p.sym ? a : 0;
    const double* A = As + r_lo * PITCH + 2 * q;
    bool ok = true;
    for (int ch = ch0; ch < nch; ++ch, ++use) {
      // in the symmetric mode's diagonal tile the products of rows 32..63 with
      // columns 0..31 are those of rows 0..31 with columns 32..63, mirrored
      const bool diag = p.sym && ch == a;
      const bool mirror = p.sym && (!diag || (wm < 2 && wn == 1));
      const int cols = t.nb - (ch * FT + wn * 32);  // of the list, in this warp's 32
      const bool idle = cols <= 0 || t.u0 + wm * 16 >= t.nb || (diag && wm >= 2 && wn == 0);
      // list columns of accumulator columns 2q + e of n8 tile nt: e * 4 + q
      int vc[4][2];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = nt * 8 + 4 * e + q;
          vc[nt][e] = !idle && c < cols ? I[ch * FT + wn * 32 + c] : -1;
        }
      const int s = use % STAGES;
      if (!wait_all(&full[s], (use / STAGES) & 1, 0x6104)) {
        ok = false;
        break;
      }
      const double* B = Bs + s * TILE + (wn * 32 + rg) * PITCH + 2 * q;
      auto release = [&] {  // the staged rows are read (the item's own with its last chunk)
        __syncwarp();
        if (lane == 0) {
          tc::mbar_arrive(&empty[s]);
          if (ch == nch - 1) tc::mbar_arrive(aempty);
        }
      };
      // the products of the warp's 16 rows with its first 8 ntv columns, into V
      auto products = [&](auto ntv) {
        constexpr int N8 = decltype(ntv)::value;
        for (int set = 0; set < t.ns; ++set) {
          const double* W = Ws + set * FT + 2 * q;
          double acc[N8][4];
#pragma unroll
          for (int nt = 0; nt < N8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0;
#pragma unroll 4
          for (int ks = 0; ks < ksteps; ++ks) {
            const double2 w = *reinterpret_cast<const double2*>(W + ks * 8);
            double2 lo = *reinterpret_cast<const double2*>(A + ks * 8);
            double2 hi = *reinterpret_cast<const double2*>(A + 8 * PITCH + ks * 8);
            double2 bv[N8];
#pragma unroll
            for (int nt = 0; nt < N8; ++nt)
              bv[nt] = *reinterpret_cast<const double2*>(B + nt * 8 * PITCH + ks * 8);
            lo.x *= w.x;
            lo.y *= w.y;
            hi.x *= w.x;
            hi.y *= w.y;
            if (ks * 8 + 8 > t.gw && ks * 8 + 2 * q >= t.gw) {  // points past the tile's end
              lo = hi = make_double2(0.0, 0.0);
#pragma unroll
              for (int nt = 0; nt < N8; ++nt) bv[nt] = make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int nt = 0; nt < N8; ++nt)
              dmma_16x8x8(acc[nt], lo.x, hi.x, lo.y, hi.y, bv[nt].x, bv[nt].y);
          }
          if (set == t.ns - 1) release();
          // V[u][v] += the products, and V[v][u] where they stand for both
          double* V = p.v + size_t(t.set0 + set) * p.v_stride;
#pragma unroll
          for (int nt = 0; nt < N8; ++nt) {
            const int vd = odd ? vc[nt][1] : vc[nt][0];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const double x0 = acc[nt][2 * h], x1 = acc[nt][2 * h + 1];
              // lane pair (g, g ^ 1): the even row's 8 columns, then the odd row's
              const double other = __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 4);
              if (vd >= 0) {
                if (u_ev[h] >= 0)
                  atomicAdd(V + size_t(u_ev[h]) * p.stride_ao + vd, odd ? other : x0);
                if (u_od[h] >= 0)
                  atomicAdd(V + size_t(u_od[h]) * p.stride_ao + vd, odd ? x1 : other);
              }
              if (mirror && u_own[h] >= 0) {
                if (vc[nt][0] >= 0) atomicAdd(V + size_t(vc[nt][0]) * p.stride_ao + u_own[h], x0);
                if (vc[nt][1] >= 0) atomicAdd(V + size_t(vc[nt][1]) * p.stride_ao + u_own[h], x1);
              }
            }
          }
        }
      };
      if (idle)
        release();
      else if (cols > 16)
        products(std::integral_constant<int, 4>());
      else
        products(std::integral_constant<int, 2>());
    }
    if (!ok) break;
  }
}

struct FockLayout {
  size_t lists, counts, items, counters, total;
};

FockLayout fock_layout(size_t nao, size_t ngrid, size_t nset, size_t blk) {
  const size_t nblk = (ngrid + blk - 1) / blk;
  const size_t gsub = (blk + FT - 1) / FT;
  const size_t max_ut = (nao + FT - 1) / FT;
  auto a256 = [](size_t x) { return (x + 255) / 256 * 256; };
  FockLayout L;
  L.lists = 0;
  L.counts = L.lists + a256(nblk * nao * sizeof(int));
  L.items = L.counts + a256(nblk * sizeof(int));
  L.counters = L.items + a256(nblk * gsub * max_ut * sizeof(int4));
  L.total = L.counters + a256(4 * sizeof(int));  // the work counter, the total, a flag
  return L;
}

}  // namespace

size_t fock_compact_workspace(size_t nao, size_t ngrid, size_t nset, size_t blk) {
  return fock_layout(nao, ngrid, nset, blk).total;
}

cudaError_t fock_compact_fp64(double* vs, const double* ws, const double* ao_lhs,
                              const double* ao_rhs, size_t stride_ao, size_t stride_grid,
                              int nao, int ngrid, int nset, const uint8_t* tab, size_t ldtab,
                              int blk, void* workspace, cudaStream_t stream) {
  if (nao <= 0 || ngrid <= 0 || nset <= 0) return cudaSuccess;
  // the work items are the AO-DM-AO kernels' 64-row, 64-point tiles
  if (aodm_row_tile() != FT || aodm_point_tile() != FT) return cudaErrorInvalidValue;
  const int nblk = (ngrid + blk - 1) / blk;
  const int gsub = (blk + FT - 1) / FT;
  const FockLayout L = fock_layout(nao, ngrid, nset, blk);
  char* wsp = static_cast<char*>(workspace);
  int* lists = reinterpret_cast<int*>(wsp + L.lists);
  int* counts = reinterpret_cast<int*>(wsp + L.counts);
  int4* items = reinterpret_cast<int4*>(wsp + L.items);
  int* counters = reinterpret_cast<int*>(wsp + L.counters);
  cudaError_t err = aodm_block_lists_launch(tab, ldtab, nao, nblk, lists, counts, stream);
  if (err != cudaSuccess) return err;
  if ((err = aodm_build_items_launch(counts, nblk, gsub, items, counters, 2, stream)) !=
      cudaSuccess)
    return err;
  FockArgs a{};
  a.v = vs;
  a.stride_ao = stride_ao;
  a.v_stride = stride_ao * stride_ao;
  a.w = ws;
  a.ao_lhs = ao_lhs;
  a.ao_rhs = ao_rhs;
  a.stride_grid = stride_grid;
  a.lists = lists;
  a.counts = counts;
  a.nao = nao;
  a.ngrid = ngrid;
  a.nset = nset;
  a.blk = blk;
  a.gsub = gsub;
  a.sym = ao_lhs == ao_rhs;
  // bulk copies need every tile's first point (b * blk + 64 t) 16-byte aligned
  // in phi and w: an even BLKSIZE and row stride, aligned bases
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  a.vec = blk % 2 == 0 && stride_grid % 2 == 0 && al16(ao_lhs) && al16(ao_rhs) && al16(ws);
  a.items = items;
  a.counters = counters;
  static_assert(2 * (FOCK_SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
  if ((err = cudaFuncSetAttribute(fock_compact_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(FOCK_SMEM))) != cudaSuccess)
    return err;
  int dev = 0, nsm = 0;
  if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return err;
  a.ctas = 2 * nsm;
  // no more CTAs than there can be items (every one draws from one counter)
  const double most = double(nblk) * gsub * ((nao + FT - 1) / FT) * nset;
  fock_compact_kernel<<<int(std::min(most, double(a.ctas))), THREADS, FOCK_SMEM, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t fock_reset_error(cudaStream_t stream) {
  static const int zero = 0;
  return cudaMemcpyToSymbolAsync(g_fock_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice,
                                 stream);
}

cudaError_t fock_read_error(int* code) {
  return cudaMemcpyFromSymbol(code, g_fock_error, sizeof(int));
}

}  // namespace cfgmm
