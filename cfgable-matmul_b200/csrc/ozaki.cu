// ozaki.cu -- FP64 GEMM emulated on the INT8 tensor cores by the Ozaki
// scheme in its Chinese-remainder form ("Ozaki scheme II": Ozaki, Uchino and
// Imamura, 2024/2025), restated here from the mathematics:
//
//   1. scaling: row i of op(A) is multiplied by 2^e_i and column j of op(B)
//      by 2^f_j and rounded to integers A', B' with |A'| <= 2^alpha,
//      |B'| <= 2^beta, where k 2^(alpha+beta) <= M/8 and M = prod m_l;
//   2. residues: A'_l = A' mods m_l, B'_l = B' mods m_l (int8) for N pairwise
//      coprime moduli m_l <= 256;
//   3. N exact INT8 GEMMs C_l = A'_l B'_l (INT32 in TMEM, gemm_i8.cu), each
//      reduced to r_l = C_l mods m_l in its epilogue;
//   4. reconstruction: C' = A'B' is the unique integer with |C'| < M/2 and
//      C' = r_l (mod m_l): C' = sum_l r_l w_l - q M with the CRT weights w_l and
//      q = round(sum_l r_l w_l / M).  Evaluated by pairs of moduli: two
//      residues make one 24-bit integer t_p (one two-way dot product), and
//      C' = sum_p t_p W_p - q M in FP64 with W_p and M in three parts, the upper
//      two with exact products and sums (< 2^53); C = C' 2^-(e_i + f_j).
//
// The only error is the rounding of A and B to alpha / beta bits relative to
// their row / column maxima; the number of moduli sets alpha and beta.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <tuple>

#include <cooperative_groups.h>

#include "gemm_i8.cuh"
#include "ozaki.cuh"
#include "side_stream.cuh"

namespace cfgmm {

namespace cg = cooperative_groups;

// Pairwise coprime moduli, largest first (256 = 2^8, 255 = 3*5*17,
// 253 = 11*23, 247 = 13*19, 217 = 7*31, the rest prime).
static const int kModuli[kMaxModuli] = {256, 255, 253, 251, 247, 241, 239, 233,
                                        229, 227, 223, 217, 211, 199, 197, 193};

namespace {

using u128 = unsigned __int128;

int bit_length(u128 v) {
  int n = 0;
  while (v) {
    ++n;
    v >>= 1;
  }
  return n;
}

long long mod_inverse(long long a, long long m) {  // a^-1 mod m, gcd(a, m) = 1
  long long t = 0, nt = 1, r = m, nr = a % m;
  while (nr) {
    const long long qq = r / nr;
    long long tmp = t - qq * nt;
    t = nt;
    nt = tmp;
    tmp = r - qq * nr;
    r = nr;
    nr = tmp;
  }
  return t < 0 ? t + m : t;
}

int ceil_log2(long long v) {
  int n = 0;
  while ((1LL << n) < v) ++n;
  return n;
}

}  // namespace

OzakiPlan ozaki_plan(int k, int nmod, int min_bits) {
  OzakiPlan p{};
  if (nmod <= 0) {
    // smallest N whose operand precision reaches min_bits
    for (nmod = 2; nmod < kMaxModuli; ++nmod) {
      OzakiPlan t = ozaki_plan(k, nmod, min_bits);
      if (t.alpha >= min_bits && t.beta >= min_bits) break;
    }
  }
  if (nmod > kMaxModuli) nmod = kMaxModuli;
  p.nmod = nmod;
  u128 M = 1;
  for (int l = 0; l < nmod; ++l) M *= u128(kModuli[l]);
  const int logM = bit_length(M) - 1;  // floor(log2 M)
  const int P = logM - 3 - ceil_log2(k > 1 ? k : 2);
  // at most 52 bits each: the FP32 residue computation is exact up to 2^52
  // op(B) takes the smaller half when P is odd: in a host call it is split once
  // for every row block of A, and at 47 bits or fewer its residues take the
  // three-digit form (the headline shape has the larger B)
  p.beta = std::min(P / 2, kOzakiMaxBits);
  p.alpha = std::min(P - P / 2, kOzakiMaxBits);
  for (int l = 0; l < nmod; ++l) {
    p.mod[l] = kModuli[l];
    p.inv_f[l] = 1.0f / float(kModuli[l]);
  }
  // parts of W_p (the largest: the last pair's, or the last modulus alone) and M:
  // sum_p |t_p| (W_p >> T1) <= 8 2^23 2^26 = 2^52, and the same of the middle parts
  int wbits = 0;
  for (int l = 0; l < nmod; l += 2)
    wbits = std::max(wbits, bit_length(M / u128(kModuli[l] * (l + 1 < nmod ? kModuli[l + 1] : 1))));
  const int T1 = std::max(0, wbits - 26), T2 = std::max(0, T1 - 26);
  auto part = [](u128 v, int from, int to) {  // bits [from, to) of v, from `from` on
    return double((v >> from) & ((u128(1) << (to - from)) - 1));
  };
  for (int l = 0; l < nmod; l += 2) {
    const long long m = kModuli[l], m2 = l + 1 < nmod ? kModuli[l + 1] : 1;
    const u128 W = M / u128(m * m2);
    // r (M / m) inv(M / m) + r' (M / m') inv(M / m') = W (m2 inv r + m inv' r') mod M
    auto coef = [&](long long mm, long long other) -> short {
      const long long inv = mod_inverse(static_cast<long long>((M / u128(mm)) % u128(mm)), mm);
      long long v = other * inv % (m * m2);
      if (2 * v > m * m2) v -= m * m2;  // least magnitude: at most m m2 / 2 < 2^15
      return short(v);
    };
    p.c[l / 2][0] = coef(m, m2);
    p.c[l / 2][1] = l + 1 < nmod ? coef(m2, m) : short(0);
    p.w1[l / 2] = double(W >> T1);
    p.w2[l / 2] = part(W, T2, T1);
    p.w3[l / 2] = part(W, 0, T2);
  }
  p.M1 = double(M >> T1);
  p.M2 = part(M, T2, T1);
  p.M3 = part(M, 0, T2);
  p.two_T1 = std::ldexp(1.0, T1);
  p.two_T12 = std::ldexp(1.0, T1 - T2);
  p.two_T21 = std::ldexp(1.0, T2 - T1);
  p.two_T2 = std::ldexp(1.0, T2);
  p.t_x = std::ldexp(1.0, T1) / double(M);
  return p;
}

namespace {

constexpr int kNonFinite = INT_MAX;  // exponent sentinel of a row holding Inf/NaN
constexpr size_t kScanBytes = size_t(40) << 20;  // operands read twice from L2, see residues_cols

// ---------------------------------------------------------------------------
// exponents: e[r] = bits - E_r with max_p |x(r,p)| < 2^E_r (0 for a zero row,
// kNonFinite for one holding Inf/NaN).  The maximum is taken over the elements'
// magnitude bits, which order as the values do and put Inf and NaN last.
// ---------------------------------------------------------------------------
template <class T>
struct Magnitude;
template <>
struct Magnitude<double> {
  using Bits = unsigned long long;
  static __device__ __forceinline__ Bits of(double x) {
    return static_cast<Bits>(__double_as_longlong(x)) & 0x7fffffffffffffffull;
  }
  static __device__ __forceinline__ double value(Bits b) {
    return __longlong_as_double(static_cast<long long>(b));
  }
};
template <>
struct Magnitude<float> {
  using Bits = unsigned;
  static __device__ __forceinline__ Bits of(float x) { return __float_as_uint(x) & 0x7fffffffu; }
  static __device__ __forceinline__ double value(Bits b) { return __uint_as_float(b); }
};

__device__ __forceinline__ int row_exponent(double amax, int bits) {
  if (!(amax <= 1.7976931348623157e308)) return kNonFinite;  // Inf or NaN
  if (amax == 0.0) return 0;
  int E;
  frexp(amax, &E);  // amax = f 2^E, f in [0.5, 1): amax < 2^E
  return bits - E;
}

// Optional mask of the masked GEMM: element (r, p) of op(B)^T takes part only
// when tab[p * ldtab + r / blk] != 0 (impl_matmul_non0tab.rs:196-207).
struct Mask {
  const uint8_t* tab;  // null: no mask
  size_t ldtab;
  int blk;
  __device__ __forceinline__ bool on(int r, int p) const {
    return !tab || tab[size_t(p) * ldtab + r / blk] != 0;
  }
};

// ---------------------------------------------------------------------------
// residues: Y[l][r][p] = rint(x(r,p) 2^e[r]) mods m_l  (int8), p < k
// The integer v (|v| <= 2^52) is written in balanced 14-bit digits:
// w = v + 2^13 (1 + 2^14 + 2^28) gives u_t = (w >> 14t) & 0x3fff (t < 3) and
// d_3 = w >> 42 with v = sum_{t<3} (u_t - 2^13) 2^14t + d_3 2^42.  With the
// symmetric c_t = 2^(14t) mods m (|c_t| <= 127) and the balanced digits
// b_t = u_t - 2^13 (formed once per element, before the modulus loop)
//   s = b_0 + b_1 c_14 + b_2 c_28 + d_3 c_42,   |s| < 2.3e6 < 2^22,
// (three FMAs per modulus, every partial sum below 2^22) is exact in FP32 and
// congruent to v.  Then q = rint(s / m) comes out exact
// from one FMA against MAGIC = 1.5 2^23 (|s| < 2^22 keeps the error of s*inv
// below 1/(2m), the least distance of s/m from a half-integer for odd m), the
// residue r = s - m q is exact, and r + MAGIC holds r in the low byte of its
// bits.  Two elements go through each packed FP32x2 instruction (sm_100).
// Modulus 256 is the low byte of v's two's complement.
// ---------------------------------------------------------------------------
using f32x2 = unsigned long long;  // two FP32 lanes in a 64-bit register

// Per modulus l (index 0 is 256, taken from the low byte): c_14, c_28, c_42,
// 1/m and -m, each in both lanes of an FP32x2 word.
struct ResidueArgs {
  int nmod;
  f32x2 c14[kMaxModuli], c28[kMaxModuli], c42[kMaxModuli], inv[kMaxModuli], nm[kMaxModuli];
  f32x2 c16[kMaxModuli], c32[kMaxModuli];  // the 16-bit digit form's 2^16, 2^32 mods m
};

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// rint(x 2^e) for a row exponent e (0 for a row holding Inf/NaN).  The power
// of two is applied as one or two exact multiplications (ldexp outside the
// normal range of the factor).
__device__ __forceinline__ double scaled_int(double x, int e) {
  if (e == kNonFinite) return 0.0;
  if (e >= -1022 && e <= 1023)
    return rint(x * __longlong_as_double(static_cast<long long>(e + 1023) << 52));
  return rint(ldexp(x, e));
}

constexpr long long kDigitBias = 8192LL * (1 + (1LL << 14) + (1LL << 28));
// 1.5 2^52 + kDigitBias: for an integer v with |v| <= 2^50, v + kRoundBias lies in
// [2^52, 2^53), where the spacing of doubles is 1, so its mantissa field holds
// w + 2^51 (w = v + kDigitBias) and the rounding that forms it is rint(v).
constexpr double kRoundBias = 6755399441055744.0 + double(kDigitBias);
// The 16-bit digit form, for |v| <= 2^47: w = v + kDigitBias16 in [0, 2^49),
// v = sum_{t<3} (u_t - 2^15) 2^16t with u_t = (w >> 16t) & 0xffff (t < 2) and
// u_2 = w >> 32, every balanced digit within [-2^15, 2^15]; then
//   s = b_0 + b_1 c_16 + b_2 c_32,  |s| <= 2^15 (1 + 2 * 127) < 2^23,
// two FMAs per modulus, exact, and |s| < 2^23 is what the quotient needs
// (|s| 2^-24 / m, the error of s * fl(1/m), stays below 1/(2m)).
constexpr long long kDigitBias16 = 32768LL * (1 + (1LL << 16) + (1LL << 32));
constexpr double kRoundBias16 = 6755399441055744.0 + double(kDigitBias16);
// The same with two digits, for |v| <= 2^30 (f32 data): w = v + 2^15 (1 + 2^16) in
// [0, 2^32) is the double's low word; s = b_0 + b_1 c_16, one FMA per modulus (f32,
// 2000 x 2000 x 3000: 173 -> 164 us the call).
constexpr double kRoundBias2x16 = 6755399441055744.0 + 32768.0 * 65537.0;

// Digit forms of write_residues8: plain (integers up to 2^52, four 14-bit
// digits), biased (up to 2^50, four 14-bit digits read off the double's bits),
// biased16 (up to 2^47, three 16-bit digits) and biased2x16 (up to 2^30, two).
enum : int { kPlain = 0, kBiased14 = 1, kBiased16 = 2, kBiased2x16 = 3 };

// The round bias of a form (0: the plain form's).
template <int kForm>
__device__ __forceinline__ constexpr double round_bias() {
  return kForm == kBiased2x16 ? kRoundBias2x16
         : kForm == kBiased16 ? kRoundBias16
         : kForm == kBiased14 ? kRoundBias
                              : 0.0;
}

// The operand element x(r, p) 2^e as the input of write_residues8: rint(x 2^e)
// (the plain form), or that integer plus the form's round bias, rounded once by
// the FMA (the biased forms).  e = kNonFinite gives 0.
template <int kForm>
__device__ __forceinline__ double scaled(double x, int e) {
  if constexpr (kForm != kPlain) {
    constexpr double bias = round_bias<kForm>();
    if (e == kNonFinite) return bias;
    if (e >= -1022 && e <= 1023)
      return fma(x, __longlong_as_double(static_cast<long long>(e + 1023) << 52), bias);
    return rint(ldexp(x, e)) + bias;
  } else {
    return scaled_int(x, e);
  }
}
template <int kForm>
__device__ __forceinline__ double scaled_zero() {
  return round_bias<kForm>();
}

// The residues of 8 consecutive elements for every modulus, 8 bytes per modulus
// plane at Y + l * plane + off (8-byte aligned).  v[] holds integers |v| <= 2^52
// (plain form) or |v| <= 2^50 (2^47, 2^30) plus the form's round bias (biased forms:
// the digits are bit fields of the double, with no conversion to a 64-bit
// integer).  The low byte of w is v's (both digit biases are multiples of 256).
template <int kForm>
__device__ __forceinline__ void write_residues8(const ResidueArgs& a, int8_t* Y, size_t plane,
                                                size_t off, const double (&v)[8]) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  f32x2 P0[4], P1[4], P2[4], P3[4];
  uint32_t lowb[2] = {0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    float u[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if constexpr (kForm == kBiased2x16) {
        // mantissa field = w + 2^51: the low word is w
        const uint32_t lo = __double2loint(v[j + h]);
        lowb[(j + h) >> 2] |= (lo & 0xffu) << (8 * ((j + h) & 3));  // modulus 256
        u[h][0] = float(int(lo & 0xffffu) - 32768);
        u[h][1] = float(int(lo >> 16) - 32768);
        u[h][2] = u[h][3] = 0.0f;
      } else if constexpr (kForm == kBiased16) {
        // mantissa field = w + 2^51: bits 0..31 are w's, bits 32..51 are (w >> 32) + 2^19
        const uint32_t lo = __double2loint(v[j + h]), hi = __double2hiint(v[j + h]);
        lowb[(j + h) >> 2] |= (lo & 0xffu) << (8 * ((j + h) & 3));  // modulus 256
        u[h][0] = float(int(lo & 0xffffu) - 32768);
        u[h][1] = float(int(lo >> 16) - 32768);
        u[h][2] = float(int(hi & 0xfffffu) - (1 << 19) - 32768);
        u[h][3] = 0.0f;
      } else if constexpr (kForm == kBiased14) {
        // mantissa field = w + 2^51: bits 0..41 are w's, bits 42..51 are (w >> 42) + 2^9
        const uint32_t lo = __double2loint(v[j + h]), hi = __double2hiint(v[j + h]);
        lowb[(j + h) >> 2] |= (lo & 0xffu) << (8 * ((j + h) & 3));  // modulus 256
        u[h][0] = float(int(lo & 0x3fffu) - 8192);
        u[h][1] = float(int((lo >> 14) & 0x3fffu) - 8192);
        u[h][2] = float(int(__funnelshift_r(lo, hi, 28) & 0x3fffu) - 8192);
        u[h][3] = float(int((hi >> 10) & 0x3ffu) - 512);
      } else {
        const long long iv = static_cast<long long>(v[j + h]);
        lowb[(j + h) >> 2] |= uint32_t(iv & 0xff) << (8 * ((j + h) & 3));  // modulus 256
        const long long w = iv + kDigitBias;
        u[h][0] = float(int(w & 0x3fff) - 8192);
        u[h][1] = float(int((w >> 14) & 0x3fff) - 8192);
        u[h][2] = float(int((w >> 28) & 0x3fff) - 8192);
        u[h][3] = float(int(w >> 42));
      }
    }
    P0[j >> 1] = pack2(u[0][0], u[1][0]);
    P1[j >> 1] = pack2(u[0][1], u[1][1]);
    P2[j >> 1] = pack2(u[0][2], u[1][2]);
    P3[j >> 1] = pack2(u[0][3], u[1][3]);
  }
  *reinterpret_cast<uint2*>(Y + off) = make_uint2(lowb[0], lowb[1]);
  const f32x2 MAG = pack2(kMagic, kMagic), NMAG = pack2(-kMagic, -kMagic);
  // unrolled: every constant is read at a fixed offset of the parameter bank
#pragma unroll
  for (int l = 1; l < kMaxModuli; ++l) {
    if (l >= a.nmod) break;
    const f32x2 INV = a.inv[l], NM = a.nm[l];
    uint32_t bits[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      f32x2 S;
      if constexpr (kForm == kBiased2x16) {
        S = fma2(P1[q], a.c16[l], P0[q]);             // s, exact
      } else if constexpr (kForm == kBiased16) {
        S = fma2(P1[q], a.c16[l], P0[q]);
        S = fma2(P2[q], a.c32[l], S);                 // s, exact
      } else {
        S = fma2(P1[q], a.c14[l], P0[q]);
        S = fma2(P2[q], a.c28[l], S);
        S = fma2(P3[q], a.c42[l], S);                 // s, exact
      }
      const f32x2 Q = add2(fma2(S, INV, MAG), NMAG);  // rint(s / m), exact
      const f32x2 R = add2(fma2(NM, Q, S), MAG);      // (s - m q) + MAGIC
      unpack2(R, bits[2 * q], bits[2 * q + 1]);
    }
    const uint32_t w0 = __byte_perm(__byte_perm(bits[0], bits[1], 0x0040),
                                    __byte_perm(bits[2], bits[3], 0x0040), 0x5410);
    const uint32_t w1 = __byte_perm(__byte_perm(bits[4], bits[5], 0x0040),
                                    __byte_perm(bits[6], bits[7], 0x0040), 0x5410);
    *reinterpret_cast<uint2*>(Y + size_t(l) * plane + off) = make_uint2(w0, w1);
  }
}

// The largest magnitude bits of row r (element (r, p) at x[r*ld + p]) by kThreads
// threads, to all of them; every thread of the CTA calls it.
template <int kThreads, class T>
__device__ __forceinline__ typename Magnitude<T>::Bits row_max(const T* __restrict__ row, int k) {
  using Mag = Magnitude<T>;
  __shared__ typename Mag::Bits red[8];
  typename Mag::Bits mx = 0;
#pragma unroll 4
  for (int p = threadIdx.x % kThreads; p < k; p += kThreads) mx = max(mx, Mag::of(row[p]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[warp] = mx;
  __syncthreads();
  const int w0 = warp / (kThreads / 32) * (kThreads / 32);
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) mx = max(mx, red[w0 + w]);
  return mx;
}

// top[r] = the largest magnitude bits of row r, a CTA per row.
template <class T>
__global__ void __launch_bounds__(256)
maxima_rows(const T* __restrict__ x, size_t ld, int k, typename Magnitude<T>::Bits* __restrict__ top) {
  const auto mx = row_max<256>(x + size_t(blockIdx.x) * ld, k);
  if (threadIdx.x == 0) top[blockIdx.x] = mx;
}

// element (r, p) at x[r*ld + p]: kThreads threads per row, 8 consecutive p each.
// kScan: they take the row's maximum first and read it again from the caches, one
// launch instead of two; operands past kScanBytes have their maxima from
// maxima_rows, whose reads then overlap the other operand's arithmetic.
template <int kForm, int kThreads, bool kScan, class T>
__global__ void __launch_bounds__(256, 5)
residues_rows(const T* __restrict__ x, size_t ld, int rows, int k, size_t kpad, int bits,
              int* __restrict__ e, int8_t* __restrict__ Y, const __grid_constant__ ResidueArgs a,
              const typename Magnitude<T>::Bits* __restrict__ top) {
  const int t = threadIdx.x % kThreads;
  const int r = blockIdx.x * (256 / kThreads) + threadIdx.x / kThreads;
  const T* row = x + size_t(min(r, rows - 1)) * ld;
  typename Magnitude<T>::Bits mx;
  if constexpr (kScan)
    mx = row_max<kThreads>(row, k);
  else
    mx = top[min(r, rows - 1)];
  if (r >= rows) return;
  const int er = row_exponent(Magnitude<T>::value(mx), bits);
  if (t == 0) e[r] = er;
  const size_t plane = size_t(rows) * kpad;
  for (int p = 8 * t; p < k; p += 8 * kThreads) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      v[j] = (p + j < k) ? scaled<kForm>(double(row[p + j]), er) : scaled_zero<kForm>();
    write_residues8<kForm>(a, Y, plane, size_t(r) * kpad + p, v);
  }
}

// The largest magnitude of each of CW adjacent r (element (r, p) at x[p*ld + r]) over
// p in [p0, p1), to every thread of the first CW of the CTA; 256 threads.
template <int CW, class T>
__device__ __forceinline__ typename Magnitude<T>::Bits
column_max(const T* __restrict__ x, size_t ld, int rows, int r0, int p0, int p1, Mask mask) {
  using Mag = Magnitude<T>;
  using Bits = typename Mag::Bits;
  __shared__ Bits red[256 / CW][CW];
  const int c = threadIdx.x % CW, pr = threadIdx.x / CW;
  Bits mx = 0;
  if (r0 + c < rows) {
    const T* col = x + r0 + c;
    if (mask.tab) {
      for (int p = p0 + pr; p < p1; p += 256 / CW)
        if (mask.on(r0 + c, p)) mx = max(mx, Mag::of(col[size_t(p) * ld]));
    } else {
#pragma unroll 8
      for (int p = p0 + pr; p < p1; p += 256 / CW) mx = max(mx, Mag::of(col[size_t(p) * ld]));
    }
  }
  red[pr][c] = mx;
  __syncthreads();
  if (threadIdx.x < CW)
#pragma unroll
    for (int w = 0; w < 256 / CW; ++w) mx = max(mx, red[w][c]);
  return mx;
}

// The maxima of a cluster's CTAs (each with a part of p), combined through
// distributed shared memory, as exponents to exps[] of every CTA.
template <int CW, class T>
__device__ __forceinline__ void cluster_exponents(typename Magnitude<T>::Bits mx, int parts,
                                                  int bits, int* exps) {
  using Mag = Magnitude<T>;
  __shared__ typename Mag::Bits part_max[CW];
  const cg::cluster_group cluster = cg::this_cluster();
  if (threadIdx.x < CW) part_max[threadIdx.x] = mx;
  cluster.sync();
  if (threadIdx.x < CW) {
    for (int s = 0; s < parts; ++s)
      mx = max(mx, *cluster.map_shared_rank(&part_max[threadIdx.x], s));
    exps[threadIdx.x] = row_exponent(Mag::value(mx), bits);
  }
  cluster.sync();  // the maxima are read, the exponents visible
}

// The maxima of op(X) alone, for the residues of large operands: top[r] (zeroed
// before) = the largest magnitude bits of element (r, p) at x[p*ld + r].  Thread per
// r, CTA = 256 r x 128 p: 79 us for 6581 x 9583 doubles, the time of reading them
// (in clusters of 8, 64 r each, 132: 1200 CTAs are a wave of 1184 and a rest).
template <class T>
__global__ void __launch_bounds__(256)
maxima_cols(const T* __restrict__ x, size_t ld, int rows, int k,
            typename Magnitude<T>::Bits* __restrict__ top, Mask mask) {
  using Mag = Magnitude<T>;
  const int r = blockIdx.x * 256 + threadIdx.x;
  const int p0 = blockIdx.y * 128, p1 = min(k, p0 + 128);
  if (r >= rows) return;
  typename Mag::Bits mx = 0;
  if (mask.tab) {
    for (int p = p0; p < p1; ++p)
      if (mask.on(r, p)) mx = max(mx, Mag::of(x[size_t(p) * ld + r]));
  } else {
#pragma unroll 8
    for (int p = p0; p < p1; ++p) mx = max(mx, Mag::of(x[size_t(p) * ld + r]));
  }
  atomicMax(top + r, mx);
}

// element (r, p) at x[p*ld + r]: CTA = CR r, a part of the tiles of CP p, transposed
// through shared memory.
// kScan: the CTAs of a cluster (the `parts` of the same r) first take their parts'
// maxima and share them, then read their tiles again, from L2: one launch instead
// of four.  That holds while x stays in L2 (1024 x 1024 x 1024: both operands 52 ->
// 30 us); at 6581 x 9583 only 18 % of the second reads hit and the kernel took 432
// us, so operands past kScanBytes have their maxima from maxima_cols.
// The tile is 16 r x 128 p with the scan (more CTAs for a small operand) and 32 r x
// 64 p without (256 bytes per row read: 295 us for the 6581 x 9583 doubles, 340 with
// 128).  Element (p, r) sits in column tile_col(p, r) of row p: a row is written as
// a permutation of its columns, and a half-warp of the read side (two r and eight
// groups of 8 p, or one r and 16) meets 16 distinct 8-byte bank pairs.
template <int CR>
__device__ __forceinline__ int tile_col(int p, int r) {
  return CR == 32 ? r ^ ((p >> 2) & 14) : r ^ ((p >> 3) & 15);
}

template <int kForm, bool kScan, class T>
__global__ void __launch_bounds__(256, 5)
residues_cols(const T* __restrict__ x, size_t ld, int rows, int k, size_t kpad, int bits,
              int* __restrict__ e, int8_t* __restrict__ Y, const __grid_constant__ ResidueArgs a,
              Mask mask, int parts, const typename Magnitude<T>::Bits* __restrict__ top) {
  constexpr int CR = kScan ? 16 : 32, CP = 2048 / CR;
  constexpr int G = CP / 8;  // groups of 8 p: G x CR units, one per thread
  __shared__ T tile[CP][CR];
  __shared__ int exps[CR];
  const int part = blockIdx.x % parts, r0 = blockIdx.x / parts * CR;
  // with the scan each CTA has a share of the tiles, without one tile
  const int ntiles = kScan ? (k + CP - 1) / CP : 0;
  const int t0 = kScan ? int((long long)part * ntiles / parts) : part;
  const int t1 = kScan ? int((long long)(part + 1) * ntiles / parts) : part + 1;
  const int c = threadIdx.x % CR, pr = threadIdx.x / CR;  // 256 / CR rows of p per pass
  const bool rin = r0 + c < rows;
  const T* col = x + r0 + c;
  if constexpr (kScan) {
    const auto mx = column_max<CR>(x, ld, rows, r0, t0 * CP, min(k, t1 * CP), mask);
    cluster_exponents<CR, T>(mx, parts, bits, exps);
    if (part == 0 && threadIdx.x < CR && rin) e[r0 + c] = exps[c];
  } else {
    if (threadIdx.x < CR) {
      exps[c] = rin ? row_exponent(Magnitude<T>::value(top[r0 + c]), bits) : 0;
      if (part == 0 && rin) e[r0 + c] = exps[c];
    }
  }
  const size_t plane = size_t(rows) * kpad;
  const int rr = threadIdx.x / G, pg = threadIdx.x % G * 8;
  for (int t = t0; t < t1; ++t) {
    const int p0 = t * CP;
    T in[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = p0 + pr + (256 / CR) * i;
      in[i] = (p < k && rin && mask.on(r0 + c, p)) ? col[size_t(p) * ld] : T(0);
    }
    __syncthreads();  // the last tile's elements are read
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = pr + (256 / CR) * i;
      tile[p][tile_col<CR>(p, c)] = in[i];
    }
    __syncthreads();
    if (r0 + rr < rows && p0 + pg < k) {
      const int er = exps[rr];
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = (p0 + pg + j < k) ? scaled<kForm>(double(tile[pg + j][tile_col<CR>(pg + j, rr)]), er)
                                 : scaled_zero<kForm>();
      write_residues8<kForm>(a, Y, plane, size_t(r0 + rr) * kpad + p0 + pg, v);
    }
  }
}

// ---------------------------------------------------------------------------
// reconstruction: C[i][j] += 2^-(e_i + f_j) * CRT(r_0..r_{N-1})
// ---------------------------------------------------------------------------
struct ReconArgs {
  int nmod;
  int vec;                      // 4 consecutive elements of C at 16-byte boundaries
  int c[kMaxModuli / 2];        // the pair's two coefficients, 16 bits each
  double w1[kMaxModuli / 2], w2[kMaxModuli / 2], w3[kMaxModuli / 2];
  double M1, M2, M3, two_T1, two_T2, two_T12, two_T21;
  double t_x;                   // 2^T1 / M (the quotient estimate)
};

// A thread rebuilds 4 consecutive C[i][j]: its residue loads (4 bytes per
// modulus plane) are all issued before the arithmetic.  Two planes' bytes of an
// element and the pair's two coefficients go through one two-way dot product,
// whose 2^23 start makes it t + 2^23 in [0, 2^24): placed in the low word of 2^52
// it is an exact double after one subtraction.  X1 = sum_p t_p w1[p] and X2 are
// exact (every partial sum at most 2^52), X3 is rounded, at 2^-53 of 2^70 for M
// near 2^111.  X1 2^T1 / M is within 2^-15 of sum_p t_p W_p / M (2^T1 / M is near
// 2^-42 and what lies below T1 adds less than 2^27 2^T1), and |C'| <= M/8 keeps
// that within 1/8 of the integer q, so q = rint of the estimate is the one of
// exact arithmetic.
//
// What it costs is instructions and the latency of the one round trip.  14 moduli,
// one conversion and two FMAs per residue -> by pairs (32 in place of 42 FP64
// operations, C in 16-byte pieces where its rows allow): 3527 x 5000 156 -> 94 us
// (0.53 GB, 81 us at the copy rate), 3527 x 9583 (odd rows of C) 287 -> 212 us.
template <int NP, class T>
__global__ void __launch_bounds__(256)
reconstruct(T* __restrict__ c, size_t ldc, int m, int n, const int8_t* __restrict__ R,
            size_t ldr, const int* __restrict__ ea, const int* __restrict__ eb,
            const __grid_constant__ ReconArgs a) {
  const int bpr = (n + 1023) / 1024;  // CTAs per row of C
  const int i = blockIdx.x / bpr;
  const int j0 = ((blockIdx.x % bpr) * 256 + threadIdx.x) * 4;
  if (j0 >= n || i >= m) return;
  const size_t plane = size_t(m) * ldr;
  // ldr is a multiple of 16 and j0 of 4: the 4 bytes at j0 lie inside row i
  const int8_t* Ri = R + size_t(i) * ldr + j0;
  uint32_t rv[2 * NP];
#pragma unroll
  for (int l = 0; l < 2 * NP; ++l)
    rv[l] = l < 2 * NP - 1 || l < a.nmod  // the last pair may be one modulus
                ? __ldg(reinterpret_cast<const uint32_t*>(Ri + size_t(l) * plane))
                : 0u;
  // C and the scales are requested with the residues (one round trip)
  T* ci = c + size_t(i) * ldc + j0;
  const bool whole = a.vec && j0 + 4 <= n;
  T c_old[4];
  int sc[4];
  if (whole) {
    if constexpr (sizeof(T) == 8) {
      *reinterpret_cast<double2*>(c_old) = *reinterpret_cast<const double2*>(ci);
      *reinterpret_cast<double2*>(c_old + 2) = *reinterpret_cast<const double2*>(ci + 2);
    } else {
      *reinterpret_cast<float4*>(c_old) = *reinterpret_cast<const float4*>(ci);
    }
    *reinterpret_cast<int4*>(sc) = __ldg(reinterpret_cast<const int4*>(eb + j0));
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      c_old[u] = j0 + u < n ? ci[u] : T(0);
      sc[u] = j0 + u < n ? __ldg(eb + j0 + u) : 0;
    }
  }
  const int ei = __ldg(ea + i);
  bool plain = ei != kNonFinite;  // every scale is a normal power of two
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const bool fin = ei != kNonFinite && sc[u] != kNonFinite;
    sc[u] = fin ? -(ei + sc[u]) : kNonFinite;
    plain = plain && sc[u] >= -1022 && sc[u] <= 1023;
  }
  constexpr double kBias = 4503599635759104.0;    // 2^52 + 2^23
  constexpr double kRound = 6755399441055744.0;   // 1.5 2^52: adding it rounds to an integer
  double X1[4], X2[4], X3[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) X1[u] = X2[u] = X3[u] = 0.0;
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const uint32_t ab = __byte_perm(rv[2 * q], rv[2 * q + 1], 0x5140);  // elements 0, 1
    const uint32_t cd = __byte_perm(rv[2 * q], rv[2 * q + 1], 0x7362);  // elements 2, 3
    const int t[4] = {
        __dp2a_lo(a.c[q], int(ab), 1 << 23), __dp2a_hi(a.c[q], int(ab), 1 << 23),
        __dp2a_lo(a.c[q], int(cd), 1 << 23), __dp2a_hi(a.c[q], int(cd), 1 << 23)};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double td = __hiloint2double(0x43300000, t[u]) - kBias;
      X1[u] = fma(td, a.w1[q], X1[u]);  // exact
      X2[u] = fma(td, a.w2[q], X2[u]);  // exact
      X3[u] = fma(td, a.w3[q], X3[u]);
    }
  }
  T out[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double q = __dsub_rn(__dadd_rn(X1[u] * a.t_x, kRound), kRound);
    double h1 = fma(-q, a.M1, X1[u]);  // exact
    double h2 = fma(-q, a.M2, X2[u]);  // exact
    const double h3 = fma(-q, a.M3, X3[u]);
    // the middle part's carry goes to the upper one (exact), so that the lower two
    // are small and C' has one rounding
    const double k = __dsub_rn(__fma_rn(h2, a.two_T21, kRound), kRound);
    h1 += k;
    h2 = fma(-k, a.two_T12, h2);
    const double cp = fma(h1, a.two_T1, fma(h2, a.two_T2, h3));
    double val;
    if (plain || (sc[u] >= -1022 && sc[u] <= 1023))  // exact scaling by a normal power of two
      val = cp * __longlong_as_double(static_cast<long long>(sc[u] + 1023) << 52);
    else if (sc[u] == kNonFinite)
      val = __longlong_as_double(0x7ff8000000000000LL);
    else
      val = ldexp(cp, sc[u]);
    out[u] = T(double(c_old[u]) + val);  // f32: rounded once
  }
  if (whole) {
    if constexpr (sizeof(T) == 8) {
      *reinterpret_cast<double2*>(ci) = *reinterpret_cast<const double2*>(out);
      *reinterpret_cast<double2*>(ci + 2) = *reinterpret_cast<const double2*>(out + 2);
    } else {
      *reinterpret_cast<float4*>(ci) = *reinterpret_cast<const float4*>(out);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j0 + u < n) ci[u] = out[u];
  }
}

template <class T, class... Args>
void launch_reconstruct(unsigned grid, cudaStream_t stream, T* c, Args... args) {
  const ReconArgs& rc = std::get<sizeof...(Args) - 1>(std::tie(args...));
  switch ((rc.nmod + 1) / 2) {
    case 1: reconstruct<1><<<grid, 256, 0, stream>>>(c, args...); break;
    case 2: reconstruct<2><<<grid, 256, 0, stream>>>(c, args...); break;
    case 3: reconstruct<3><<<grid, 256, 0, stream>>>(c, args...); break;
    case 4: reconstruct<4><<<grid, 256, 0, stream>>>(c, args...); break;
    case 5: reconstruct<5><<<grid, 256, 0, stream>>>(c, args...); break;
    case 6: reconstruct<6><<<grid, 256, 0, stream>>>(c, args...); break;
    case 7: reconstruct<7><<<grid, 256, 0, stream>>>(c, args...); break;
    default: reconstruct<8><<<grid, 256, 0, stream>>>(c, args...); break;
  }
}

// ---------------------------------------------------------------------------
// tensor maps
// ---------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

// Planes of `rows` rows of `cols` bytes at stride `pitch`, boxes of 128 bytes x
// box_rows rows, 128-byte swizzle.
bool make_plane_map(CUtensorMap* map, void* base, int cols, int rows, int nplanes, size_t pitch,
                    int box_rows) {
  auto enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[3] = {cuuint64_t(cols), cuuint64_t(rows), cuuint64_t(nplanes)};
  cuuint64_t strides[2] = {cuuint64_t(pitch), cuuint64_t(rows) * pitch};
  cuuint32_t box[3] = {128, cuuint32_t(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

size_t a256(size_t v) { return (v + 255) / 256 * 256; }

struct DgemmLayout {
  size_t kpad, ldr, a_res, b_res, r, ea, eb, top_a, top_b, total;
};

DgemmLayout dgemm_layout(int m, int n, int k, int nmod) {
  DgemmLayout L;
  L.kpad = (size_t(k) + 127) / 128 * 128;
  L.ldr = (size_t(n) + 15) / 16 * 16;
  L.a_res = 0;
  L.b_res = L.a_res + a256(size_t(nmod) * m * L.kpad);
  L.r = L.b_res + a256(size_t(nmod) * n * L.kpad);
  L.ea = L.r + a256(size_t(nmod) * m * L.ldr);
  L.eb = L.ea + a256(size_t(m) * sizeof(int));
  L.top_a = L.eb + a256(size_t(n) * sizeof(int));
  L.top_b = L.top_a + a256(size_t(m) * sizeof(double));
  L.total = L.top_b + a256(size_t(n) * sizeof(double));
  return L;
}

int mods_host(long long v, int m) {  // symmetric residue
  long long r = v % m;
  if (r < 0) r += m;
  if (r > (m - 1) / 2) r -= m;
  return int(r);
}

// both FP32 lanes of a packed word set to v
f32x2 splat2(float v) {
  uint32_t b;
  std::memcpy(&b, &v, sizeof b);
  return (f32x2(b) << 32) | b;
}

ResidueArgs residue_args(const OzakiPlan& p) {
  ResidueArgs a{};
  a.nmod = p.nmod;
  for (int l = 0; l < p.nmod; ++l) {
    a.inv[l] = splat2(p.inv_f[l]);
    a.nm[l] = splat2(-float(p.mod[l]));
    a.c14[l] = splat2(float(mods_host(1LL << 14, p.mod[l])));
    a.c28[l] = splat2(float(mods_host(1LL << 28, p.mod[l])));
    a.c42[l] = splat2(float(mods_host(1LL << 42, p.mod[l])));
    a.c16[l] = splat2(float(mods_host(1LL << 16, p.mod[l])));
    a.c32[l] = splat2(float(mods_host(1LL << 32, p.mod[l])));
  }
  return a;
}

template <int kForm, class T>
cudaError_t prepare_form(const T* x, size_t ld, bool rows_contig, int rows, int k, size_t kpad,
                         int bits, void* top, int* e, int8_t* Y, const ResidueArgs& ra,
                         cudaStream_t s, Mask mask) {
  using Bits = typename Magnitude<T>::Bits;
  Bits* maxima = static_cast<Bits*>(top);
  bool scan = size_t(rows) * k * sizeof(T) <= kScanBytes;
  if (rows_contig) {
    if (!scan) {
      maxima_rows<T><<<rows, 256, 0, s>>>(x, ld, k, maxima);
      residues_rows<kForm, 256, false, T>
          <<<rows, 256, 0, s>>>(x, ld, rows, k, kpad, bits, e, Y, ra, maxima);
    } else if (k <= 512) {  // short rows share a CTA
      residues_rows<kForm, 64, true, T>
          <<<(rows + 3) / 4, 256, 0, s>>>(x, ld, rows, k, kpad, bits, e, Y, ra, nullptr);
    } else {
      residues_rows<kForm, 256, true, T>
          <<<rows, 256, 0, s>>>(x, ld, rows, k, kpad, bits, e, Y, ra, nullptr);
    }
    return cudaGetLastError();
  }
  // Few rows over a long k: the scan's clusters are few and walk many tiles each, one
  // after the other.  Both operands by columns, us the call with the scan / without:
  // 64 x 64 x 60000 (59 tiles to a CTA) 370 / 220, 200 x 200 x 16000 131 / 118, 30 x 30 x
  // 13000 (13 tiles) 78 / 61, 500 x 500 x 13000 in f32 126 / 120.
  if ((rows + 15) / 16 * 8 < 592 && k > 8 * 12 * 128) scan = false;
  int parts = 8;
  while (parts > (k + 127) / 128) parts /= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned((rows + 15) / 16) * parts);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = unsigned(parts);
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (scan)
    return cudaLaunchKernelEx(&cfg, residues_cols<kForm, true, T>, x, ld, rows, k, kpad, bits, e,
                              Y, ra, mask, parts, static_cast<const Bits*>(nullptr));
  cudaError_t err = cudaMemsetAsync(maxima, 0, size_t(rows) * sizeof(Bits), s);
  if (err != cudaSuccess) return err;
  maxima_cols<T><<<dim3((rows + 255) / 256, (k + 127) / 128), 256, 0, s>>>(x, ld, rows, k, maxima,
                                                                          mask);
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  const int ntiles = (k + 63) / 64;
  residues_cols<kForm, false, T><<<unsigned((rows + 31) / 32) * ntiles, 256, 0, s>>>(
      x, ld, rows, k, kpad, bits, e, Y, ra, mask, ntiles, maxima);
  return cudaGetLastError();
}

// Scales, rounds and splits op(X) into residue planes Y[nmod][rows][kpad], the
// rows' exponents into e; `top` is scratch for rows doubles.
template <class T>
cudaError_t prepare(const T* x, size_t ld, bool rows_contig, int rows, int k, size_t kpad,
                    int bits, void* top, int* e, int8_t* Y, const ResidueArgs& ra, cudaStream_t s,
                    Mask mask = Mask{nullptr, 0, 1}) {
  // scaled elements up to 2^30 take two 16-bit digits, up to 2^47 three, up to
  // 2^50 the biased form of four 14-bit digits, the rest the plain form
  if (bits <= 30)
    return prepare_form<kBiased2x16>(x, ld, rows_contig, rows, k, kpad, bits, top, e, Y, ra, s,
                                     mask);
  if (bits <= 47)
    return prepare_form<kBiased16>(x, ld, rows_contig, rows, k, kpad, bits, top, e, Y, ra, s, mask);
  if (bits <= 50)
    return prepare_form<kBiased14>(x, ld, rows_contig, rows, k, kpad, bits, top, e, Y, ra, s, mask);
  return prepare_form<kPlain>(x, ld, rows_contig, rows, k, kpad, bits, top, e, Y, ra, s, mask);
}

}  // namespace

const SideStream* side_stream(bool high_priority) {
  constexpr int kMaxDevices = 64;
  thread_local SideStream streams[kMaxDevices][2];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  SideStream& st = streams[dev][high_priority ? 1 : 0];
  if (!st.join) {
    // made in place; a partial set (one creation failed) is kept, released at
    // thread exit, and completed by a later call
    int lo = 0, hi = 0;
    if (high_priority && cudaDeviceGetStreamPriorityRange(&lo, &hi) != cudaSuccess) return nullptr;
    if (!st.s && cudaStreamCreateWithPriority(&st.s, cudaStreamNonBlocking, high_priority ? hi : 0) !=
                     cudaSuccess) {
      st.s = nullptr;
      return nullptr;
    }
    if (!st.fork && cudaEventCreateWithFlags(&st.fork, cudaEventDisableTiming) != cudaSuccess) {
      st.fork = nullptr;
      return nullptr;
    }
    if (cudaEventCreateWithFlags(&st.join, cudaEventDisableTiming) != cudaSuccess) {
      st.join = nullptr;
      return nullptr;
    }
  }
  return &st;
}


int ozaki_default_moduli(int k) {
  const char* env = std::getenv("CFGMM_OZAKI_MODULI");
  if (env) {
    const int v = std::atoi(env);
    if (v >= 2 && v <= kMaxModuli) return v;
  }
  return ozaki_plan(k, 0, kOzakiMinBits).nmod;
}

int ozaki_moduli_for_bits(int k, int bits) { return ozaki_plan(k, 0, bits).nmod; }

size_t ozaki_dgemm_workspace(int m, int n, int k, int nmod) {
  return dgemm_layout(m, n, k, nmod).total;
}

template <class T>
cudaError_t ozaki_dgemm(T* c, const T* a, const T* b, int m, int n, int k,
                        size_t lda, size_t ldb, size_t ldc, bool transa, bool transb, int nmod,
                        void* workspace, cudaStream_t stream, const cudaEvent_t* events,
                        const uint8_t* tab, size_t ldtab, int blk, cudaEvent_t c_ready,
                        int m_layout, int n_layout, bool reuse_a, bool reuse_b) {
  if (tab && transb) return cudaErrorInvalidValue;  // the masked GEMM has no transb
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  auto mark = [&](int i) { if (events) cudaEventRecord(events[i], stream); };
  if (k > kOzakiMaxK) return cudaErrorInvalidValue;
  const OzakiPlan plan = ozaki_plan(k, nmod, 0);
  if (m_layout < m) m_layout = m;
  if (n_layout < n) n_layout = n;
  const DgemmLayout L = dgemm_layout(m_layout, n_layout, k, plan.nmod);
  char* ws = static_cast<char*>(workspace);
  int8_t* a_res = reinterpret_cast<int8_t*>(ws + L.a_res);
  int8_t* b_res = reinterpret_cast<int8_t*>(ws + L.b_res);
  int8_t* r = reinterpret_cast<int8_t*>(ws + L.r);
  int* ea = reinterpret_cast<int*>(ws + L.ea);
  int* eb = reinterpret_cast<int*>(ws + L.eb);
  const ResidueArgs ra = residue_args(plan);
  mark(0);
  // op(A) rows are i (k contiguous unless transa); op(B) "rows" are j
  // (k contiguous only when transb).
  cudaError_t err = cudaSuccess;
  // With both operands to prepare, one's kernel runs on a side stream beside the other's:
  // their phases are bound by instruction issue (residues) and by memory (the
  // scan for the exponents), so the two overlap.  The side stream joins back before the
  // GEMM (the fork and join are events, so a stream capture follows them).  The side
  // stream starts later, and an operand by rows goes there: clusters of an operand by
  // columns that start behind its CTAs share fewer SMs.  A by columns with B by rows, us
  // with B / A on the side: 300 x 300 x 6000 63 / 97, 200 x 200 x 3000 36 / 59, 1500 x 700
  // x 2500 100 / 121, 2000 x 2000 x 2000 in f32 123 / 133; A by rows with B by columns
  // the other way round; two of one kind alike.
  SideScope side((!reuse_a && !reuse_b) ? side_stream() : nullptr, stream);
  if ((err = side.fork()) != cudaSuccess) return err;
  const bool b_aside = transa && transb;
  const cudaStream_t sa = b_aside ? stream : side.stream(), sb = b_aside ? side.stream() : stream;
  if (!reuse_a) {
    err = prepare(a, lda, !transa, m, k, L.kpad, plan.alpha, ws + L.top_a, ea,
                  a_res, ra, sa);
    if (err != cudaSuccess) return err;
  }
  if (!reuse_b) {
    err = prepare(b, ldb, transb, n, k, L.kpad, plan.beta, ws + L.top_b, eb, b_res, ra, sb,
                  Mask{tab, ldtab, blk > 0 ? blk : 1});
    if (err != cudaSuccess) return err;
  }
  if ((err = side.join()) != cudaSuccess) return err;

  mark(1);
  CUtensorMap tmA, tmB, tmR;
  if (!make_plane_map(&tmR, r, n, m, plan.nmod, L.ldr, 32) ||
      !make_plane_map(&tmA, a_res, k, m, plan.nmod, L.kpad, gemm_i8_tile_rows_a()) ||
      !make_plane_map(&tmB, b_res, k, n, plan.nmod, L.kpad, gemm_i8_tile_rows_b()))
    return cudaErrorInvalidValue;
  GemmI8Args g{};
  g.rows_a = m;
  g.rows_b = n;
  g.k = k;
  g.nmod = plan.nmod;
  g.out = r;
  g.ldr = L.ldr;
  for (int l = 0; l < plan.nmod; ++l) {
    g.mod[l] = plan.mod[l];
    g.mul[l] = int((2 * (1ll << 38) / plan.mod[l] + 1) / 2);  // rint(2^38 / mod)
  }
  if ((err = gemm_i8_mod(tmA, tmB, tmR, g, stream)) != cudaSuccess) return err;
  mark(2);

  ReconArgs rc{};
  rc.nmod = plan.nmod;
  for (int q = 0; q < (plan.nmod + 1) / 2; ++q) {
    rc.c[q] = int(uint32_t(uint16_t(plan.c[q][0])) | uint32_t(uint16_t(plan.c[q][1])) << 16);
    rc.w1[q] = plan.w1[q];
    rc.w2[q] = plan.w2[q];
    rc.w3[q] = plan.w3[q];
  }
  rc.M1 = plan.M1;
  rc.M2 = plan.M2;
  rc.M3 = plan.M3;
  rc.two_T1 = plan.two_T1;
  rc.two_T12 = plan.two_T12;
  rc.two_T21 = plan.two_T21;
  rc.two_T2 = plan.two_T2;
  rc.t_x = plan.t_x;
  rc.vec = reinterpret_cast<uintptr_t>(c) % 16 == 0 && ldc * sizeof(T) % 16 == 0;
  const long long rgrid = (long long)((n + 1023) / 1024) * m;
  if (rgrid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  if (c_ready && (err = cudaStreamWaitEvent(stream, c_ready, 0)) != cudaSuccess) return err;
  launch_reconstruct(unsigned(rgrid), stream, c, ldc, m, n, r, L.ldr, ea, eb, rc);
  mark(3);
  return cudaGetLastError();
}

template cudaError_t ozaki_dgemm<double>(double*, const double*, const double*, int, int, int,
                                         size_t, size_t, size_t, bool, bool, int, void*,
                                         cudaStream_t, const cudaEvent_t*, const uint8_t*, size_t,
                                         int, cudaEvent_t, int, int, bool, bool);
template cudaError_t ozaki_dgemm<float>(float*, const float*, const float*, int, int, int, size_t,
                                        size_t, size_t, bool, bool, int, void*, cudaStream_t,
                                        const cudaEvent_t*, const uint8_t*, size_t, int,
                                        cudaEvent_t, int, int, bool, bool);

}  // namespace cfgmm
