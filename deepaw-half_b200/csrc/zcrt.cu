// Complex FP64 products on the int8 tensor cores (tcgen05 kind::i8) by the
// Chinese remainder theorem, for large products of a mixed solve's FP64 phase.
//
// The B200's FP64 pipes give about 37 TFLOP/s, vector or tensor, and ZGEMM
// runs at that rate on the large cells, so a faster product has to leave
// them.  Method (Ozaki, Uchino and Imamura, "Ozaki scheme II", 2025): every
// row of op(A) and column of op(B) is scaled by a power of two to a norm
// below 2^62 and rounded to integers; the integer product is formed modulo 16
// coprime moduli p_i <= 256, each an int8 product with exact int32
// accumulation, and put together again.  By Cauchy-Schwarz the integer sums
// are below 2^124, inside half the moduli's product of 2^125.4, so the result
// is exact up to the rounding of the operands: an element is held in units of
// at most 2^-61 of its row's norm, full FP64 down to 2^-9 of that norm and
// fewer bits below.  The error of an element of the product is at most
// 2 sqrt(K) 2^-61.5 |a| |b| and a rounding of the result; measured, 2^-60 |a| |b|.
//
// That bound is relative to the norms, where ZGEMM's is relative to
// sum |a_k| |b_k|.  So the product is for operands whose rows are not graded
// against each other, and a caller has to allow it: the iteration does for its
// projections, its S-orthogonalisation and the projector products, in the
// FP64 phase of a mixed solve only, and not for its rotations and pencils.
// Errors there against double-double sums, beside ZGEMM's on the same
// operands (rms over 4,096 elements and every iteration; worst product):
// relative to |a| |b|, 0.02 of ZGEMM's for the projectors' B^H X, 0.02 for
// X^H S P, 0.09 for the projections, and equal (the rounding of the sum it is
// added to) for the two that accumulate; relative to sum |a_k| |b_k|, 0.02,
// 0.02, 0.1, 0.94 and 0.98 (216-atom cell, 480 bands, 2e-5 and 1e-7 eV), and
// 0.2 to 0.7 on the 12-atom cell with 512 bands to 1e-9 eV.  (The rotations,
// with the columns of [X P] scaled alike, would be at 0.07 and 900.)  Where
// translational symmetry makes vectors' supports disjoint (64-atom cell, no
// atom displaced), ZGEMM leaves the elements that vanish by it at zero, and
// they are about 2^-61 |a| |b| here; relative to |a| |b| the worst is 0.12.
//
//   crt_norm_*      row norms -> power-of-two scales
//   crt_split       residues of Re and Im, 32 bytes per element, in the
//                   K-major no-swizzle UMMA layout: 8 rows x 128 k are 1 KB
//                   (8 core matrices of 8 rows x 16 bytes), so a stage's tile
//                   of one plane is one contiguous bulk copy
//   crt_gemm_kernel one CTA per (128 x kBN tile, modulus): one thread issues
//                   the copies, one the MMAs (Ar Br, Ai Bi, and Ar Bi + Ai Br
//                   into three int32 TMEM accumulators), eight warps reduce
//                   the sums modulo p and store one byte per part
//   crt_join        x / P = frac(sum_i r_i y_i / p_i) in 96-bit fixed point,
//                   times P and the scales
//
// The product is bound by the tensor pipe (82 % of its cycles on 600 x 600 x
// 38,089: 0.64 ms; three accumulators leave one CTA per SM, whose start and
// epilogue are the rest), the split by its integer dot products (0.40 ms an
// operand, the norms 0.07).  Both operands split, one product, ZGEMM / this:
// X^H Y 600 x 600 x 38,089 3.22 / 1.61 ms, upper half of 1,200 x 1,200 x 38,089
// 12.5 / 3.4 ms (ZGEMM of the whole matrix), 1,696 x 600 x 38,089 8.91 / 3.49
// ms, X C 38,089 x 600 x 600 3.16 / 2.23 ms.
#include <algorithm>
#include <climits>
#include <cmath>

#include "tc.cuh"
#include "tc_gemm.h"
#include "zcrt.h"

namespace hb {

namespace {

using namespace tc;

constexpr int kMods = 16;
constexpr int kScaleBits = 62;     // row norms are scaled below 2^62; the sums stay below 2^124 < P / 2 = 2^124.4
constexpr int kMod[kMods] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
constexpr int kMaxK = 65000;       // |2 K 128 128| < 2^31
constexpr int kBM = 128, kBN = 160;   // three int32 accumulators of kBN columns fit Tensor Memory
constexpr int kKB = 128;           // k per stage
constexpr int kStages = 3;
constexpr uint32_t kAPlane = kBM * kKB, kBPlane = kBN * kKB;       // bytes of one plane's tile
constexpr uint32_t kStage = 2 * (kAPlane + kBPlane);
constexpr int kThreads = 10 * 32;
constexpr size_t kSmem = size_t(kStages) * kStage + 1024;
constexpr int kNaN = INT_MIN;      // scale of a row that holds a NaN or an infinity

struct Modulus {
  int p;
  unsigned magic;        // floor(2^32 / p) + 1
  int wlo, whi;          // 2^(8 j) mod p, balanced, as packed signed bytes
  int bias;              // makes the split's weighted byte sum positive and undoes its 2^62 offset
  unsigned bias32;       // multiple of p just above 2^31
  unsigned long long fhi;   // y / p with y = (P / p)^-1 mod p, as a 96-bit fraction
  unsigned flo;
};
struct Moduli {
  Modulus m[kMods];
  double phi, plo;       // P 2^-64 as a pair
};

int mod_pow2(int bits, int p) {
  int r = 1 % p;
  for (int i = 0; i < bits; ++i) r = 2 * r % p;
  return r;
}

const Moduli& moduli() {
  static const Moduli table = [] {
    Moduli t{};
    unsigned __int128 P = 1;
    for (int i = 0; i < kMods; ++i) P *= unsigned(kMod[i]);
    for (int i = 0; i < kMods; ++i) {
      Modulus& m = t.m[i];
      const int p = m.p = kMod[i];
      m.magic = unsigned((1ull << 32) / unsigned(p)) + 1u;
      unsigned w[2] = {0, 0};
      for (int j = 0; j < 8; ++j) {
        int r = mod_pow2(8 * j, p);
        if (r > 127) r -= p;
        w[j / 4] |= unsigned(r & 255) << (8 * (j % 4));
      }
      m.wlo = int(w[0]);
      m.whi = int(w[1]);
      m.bias = p * ((8 * 255 * 128 + p - 1) / p) + (p - mod_pow2(62, p)) % p;
      m.bias32 = unsigned(((1ull << 31) + unsigned(p) - 1) / unsigned(p) * unsigned(p));
      const int q = int(P / unsigned(p) % unsigned(p));
      int y = 1 % p;
      while ((long long)q * y % p != 1 % p) ++y;
      const unsigned __int128 num = (unsigned __int128)unsigned(y) << 64;
      m.fhi = (unsigned long long)(num / unsigned(p));
      m.flo = unsigned(((unsigned long long)(num % unsigned(p)) << 32) / unsigned(p));
    }
    const double hi = double((unsigned long long)(P >> 64)) * 0x1p64;
    const double ph = hi + double((unsigned long long)P);   // P rounded
    const __int128 rest = (__int128)P - (__int128)((unsigned __int128)(ph * 0x1p-57) << 57);   // ph is a multiple of 2^57
    t.phi = ph * 0x1p-64;
    t.plo = double(rest) * 0x1p-64;
    return t;
  }();
  return table;
}

__device__ __forceinline__ const double2* row_of(const CrtSide& s, int r) {   // k contiguous
  return r < s.split ? s.p + (long long)r * s.ld : s.p2 + (long long)(r - s.split) * s.ld;
}
__device__ __forceinline__ const double2* column_of(const CrtSide& s, int k) {   // rows contiguous
  return k < s.split ? s.p + (long long)k * s.ld : s.p2 + (long long)(k - s.split) * s.ld;
}

// Scale of a row from the sum of squares and the largest part's magnitude.
__device__ int scale_of(double sum, double big, int k) {
  if (!isfinite(big)) return kNaN;
  if (big == 0.0) return 0;
  // squares that overflowed or went subnormal: bound the norm by the largest part
  const double norm = sum < 1e300 && sum > 1e-280 ? sqrt(sum) * (1.0 + 1e-10) : 0.0;
  const int ex = norm > 0.0 ? ilogb(norm) + 1 : ilogb(big) + 2 + (33 - __clz(k)) / 2;
  return kScaleBits - ex;
}

// max that keeps a NaN or infinity visible
__device__ __forceinline__ double big_of(double b, double2 v) {
  const double m = fmax(fabs(v.x), fabs(v.y));
  return isfinite(v.x) && isfinite(v.y) ? fmax(b, m) : HUGE_VAL;
}

__global__ void __launch_bounds__(256) crt_norm_k(CrtSide s, int* __restrict__ e) {
  const int r = blockIdx.x;
  const double2* p = row_of(s, r);
  double sum = 0.0, big = 0.0;
  for (int k = threadIdx.x; k < s.k; k += 256) {
    const double2 v = p[k];
    sum += v.x * v.x + v.y * v.y;
    big = big_of(big, v);
  }
  __shared__ double ss[8], sb[8];
  for (int off = 16; off > 0; off >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, off);
    big = fmax(big, __shfl_xor_sync(0xffffffffu, big, off));
  }
  if ((threadIdx.x & 31) == 0) {
    ss[threadIdx.x >> 5] = sum;
    sb[threadIdx.x >> 5] = big;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      sum += ss[w];
      big = fmax(big, sb[w]);
    }
    e[r] = scale_of(sum, big, s.k);
  }
}

// 64 rows per CTA, four threads per row
__global__ void __launch_bounds__(256) crt_norm_mn(CrtSide s, int* __restrict__ e) {
  const int rl = threadIdx.x & 63, part = threadIdx.x >> 6, r = blockIdx.x * 64 + rl;
  double sum = 0.0, big = 0.0;
  if (r < s.rows)
    for (int k = part; k < s.k; k += 4) {
      const double2 v = column_of(s, k)[r];
      sum += v.x * v.x + v.y * v.y;
      big = big_of(big, v);
    }
  __shared__ double ss[4][64], sb[4][64];
  ss[part][rl] = sum;
  sb[part][rl] = big;
  __syncthreads();
  if (part == 0 && r < s.rows) {
    for (int w = 1; w < 4; ++w) {
      sum += ss[w][rl];
      big = fmax(big, sb[w][rl]);
    }
    e[r] = scale_of(sum, big, s.k);
  }
}

__device__ __forceinline__ int dot4_us(unsigned bytes, int weights, int acc) {
  int r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(bytes), "r"(weights), "r"(acc));
  return r;
}

// balanced residue (a signed byte) of the integer held as u = q + 2^62
__device__ __forceinline__ int residue(unsigned long long u, const Modulus& m) {
  const int v = dot4_us(unsigned(u), m.wlo, dot4_us(unsigned(u >> 32), m.whi, m.bias));
  int r = v - int(__umulhi(unsigned(v), m.magic)) * m.p;
  return r > 127 ? r - m.p : r;
}

__device__ __forceinline__ unsigned long long to_integer(double x, double s1, double s2) {
  return (unsigned long long)__double2ll_rn(x * s1 * s2) + (1ull << 62);   // |x s1 s2| <= 2^62
}

// Planes of a side: part q of modulus i at out + (2 i + q) plane_bytes; element
// (r, k) of a plane at (k / 128) rows_pad 128 + (r / 8) 1024 + (k % 128 / 16) 128
// + (r % 8) 16 + k % 16.  A warp takes 8 rows x 16 k, a lane one row and four
// consecutive k, so that each store of a warp fills one core matrix.
template <bool KC>
__global__ void __launch_bounds__(256) crt_split(CrtSide s, const int* __restrict__ e, Moduli mods, int rows_pad,
                                                 int k_pad, unsigned char* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const long long w = blockIdx.x * 8ll + (threadIdx.x >> 5);
  const int kc = k_pad / 16;
  const long long rg = w / kc;
  const int chunk = int(w - rg * kc);
  if (rg >= rows_pad / 8) return;
  const int r = int(rg) * 8 + (lane >> 2), k0 = chunk * 16 + (lane & 3) * 4;
  const bool row_on = r < s.rows;
  const int ex = row_on ? e[r] : 0;
  // 2^ex as two factors, each in range for every double
  const double s1 = ex == kNaN ? 0.0 : scalbn(1.0, ex / 2), s2 = ex == kNaN ? 0.0 : scalbn(1.0, ex - ex / 2);
  unsigned long long re[4], im[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double2 v = make_double2(0.0, 0.0);
    if (row_on && ex != kNaN && k0 + i < s.k) {
      v = KC ? row_of(s, r)[k0 + i] : column_of(s, k0 + i)[r];
      if (s.conj) v.y = -v.y;
    }
    re[i] = to_integer(v.x, s1, s2);
    im[i] = to_integer(v.y, s1, s2);
  }
  const long long plane = (long long)rows_pad * k_pad;
  unsigned char* o = out + (long long)(chunk >> 3) * rows_pad * 128 + rg * 1024 + (chunk & 7) * 128 + (lane >> 2) * 16 +
                     (lane & 3) * 4;
#pragma unroll
  for (int i = 0; i < kMods; ++i) {
    const Modulus& m = mods.m[i];
    unsigned a = 0, b = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a |= unsigned(residue(re[j], m) & 255) << (8 * j);
      b |= unsigned(residue(im[j], m) & 255) << (8 * j);
    }
    *reinterpret_cast<unsigned*>(o + (2 * i) * plane) = a;
    *reinterpret_cast<unsigned*>(o + (2 * i + 1) * plane) = b;
  }
}

// kind::i8 instruction descriptor: signed 8-bit operands, 32-bit integer sums, M = 128.
constexpr uint32_t kDescI8 =
    (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kBN >> 3) << 17) | (uint32_t(kBM >> 4) << 24);

__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, bool accumulate) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(kDescI8), "r"(uint32_t(accumulate)), "r"(z), "r"(z), "r"(z), "r"(z));
}

// x mod p in [0, p)
__device__ __forceinline__ int reduce(int x, const Modulus& m) {
  const unsigned u = unsigned(x) + m.bias32;
  const int r = int(u - __umulhi(u, m.magic) * unsigned(m.p));   // the quotient may be one too large
  return r < 0 ? r + m.p : r;
}

// res: part q of modulus i of slice s at ((2 (s kMods + i) + q) N + col) m_pad + row, one byte each.
__global__ void __launch_bounds__(kThreads, 1)
    crt_gemm_kernel(const unsigned char* __restrict__ A, const unsigned char* __restrict__ B, int a_rows_pad,
                    int b_rows_pad, int k_pad, int steps_per, int N, int m_pad, bool upper, Moduli mods,
                    unsigned char* __restrict__ res, int* err) {
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  __shared__ uint64_t full_bar[kStages], empty_bar[kStages], accum_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN, slice = blockIdx.z / kMods, mod = blockIdx.z % kMods;
  if (upper && m0 >= n0 + kBN) return;   // wholly below the diagonal
  const uint32_t sbase = (smem_addr(smem_dyn) + 1023u) & ~1023u;
  const int i0 = slice * steps_per, steps = min(k_pad / kKB - i0, steps_per);   // this slice of K
  volatile int* abort = &abort_flag;
  if (warp == 9) tmem_alloc(&tmem_slot, 512);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&accum_bar, 1);
    abort_flag = 0;
    mbar_init_fence();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  const long long a_plane = (long long)a_rows_pad * k_pad, b_plane = (long long)b_rows_pad * k_pad;
  if (warp == 8) {
    if (lane == 0) {
      int issued = 0;
      for (int i = 0; i < steps; ++i) {
        const int s = i % kStages;
        if (i >= kStages && !mbar_wait(&empty_bar[s], ((i / kStages) - 1) & 1, abort)) break;
        const uint32_t base = sbase + uint32_t(s) * kStage;
        mbar_expect_tx(&full_bar[s], kStage);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          bulk_copy_g2s(base + q * kAPlane, A + (2 * mod + q) * a_plane + ((long long)(i0 + i) * a_rows_pad + m0) * kKB, kAPlane,
                        &full_bar[s]);
          bulk_copy_g2s(base + 2 * kAPlane + q * kBPlane,
                        B + (2 * mod + q) * b_plane + ((long long)(i0 + i) * b_rows_pad + n0) * kKB, kBPlane, &full_bar[s]);
        }
        mbar_arrive(&full_bar[s]);
        issued = i + 1;
      }
      if (*abort) {   // let the copies still in flight land before the CTA leaves
        for (int i = max(0, issued - kStages); i < issued; ++i) mbar_wait_drain(&full_bar[i % kStages], (i / kStages) & 1);
      }
    }
  } else if (warp == 9) {
    if (lane == 0) {
      for (int i = 0; i < steps; ++i) {
        const int s = i % kStages;
        if (!mbar_wait(&full_bar[s], (i / kStages) & 1, abort)) break;
        tcgen05_fence_after();
        const uint32_t a0 = sbase + uint32_t(s) * kStage, b0 = a0 + 2 * kAPlane;
#pragma unroll
        for (int q = 0; q < kKB / 32; ++q) {
          const uint64_t ar = smem_desc(a0 + q * 256u, 128u, 1024u), ai = smem_desc(a0 + kAPlane + q * 256u, 128u, 1024u);
          const uint64_t br = smem_desc(b0 + q * 256u, 128u, 1024u), bi = smem_desc(b0 + kBPlane + q * 256u, 128u, 1024u);
          const bool more = i > 0 || q > 0;
          mma_i8(tmem, ar, br, more);
          mma_i8(tmem + kBN, ai, bi, more);
          mma_i8(tmem + 2 * kBN, ar, bi, more);
          mma_i8(tmem + 2 * kBN, ai, br, true);
        }
        mma_commit(&empty_bar[s]);
      }
      mma_commit(&accum_bar);   // also on abort: arrives once every issued MMA has completed
    }
  } else {
    const bool done = __all_sync(0xffffffffu, mbar_wait_drain(&accum_bar, 0));
    if (done && !*abort) {
      tcgen05_fence_after();
      const Modulus m = mods.m[mod];
      const int q = warp & 3, half = warp >> 2;
      const int row = m0 + q * 32 + lane;
      unsigned char* o_re = res + (long long)(2 * (slice * kMods + mod)) * N * m_pad + row;
      unsigned char* o_im = o_re + (long long)N * m_pad;
      for (int c = half; c < kBN / 8; c += 2) {
        float t1[8], t2[8], t3[8];   // bit patterns of the integer sums
        const uint32_t ta = tmem + (uint32_t(q * 32) << 16) + uint32_t(c * 8);
        tmem_ld8(ta, t1);
        tmem_ld8(ta + kBN, t2);
        tmem_ld8(ta + 2 * kBN, t3);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = n0 + c * 8 + j;
          if (col >= N) break;
          o_re[(long long)col * m_pad] = (unsigned char)reduce(__float_as_int(t1[j]) - __float_as_int(t2[j]), m);
          o_im[(long long)col * m_pad] = (unsigned char)reduce(__float_as_int(t3[j]), m);
        }
      }
    } else if (!done) {
      *abort = 1;
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 9) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(err, 1);
}

// C = alpha x + beta C from the residues.  A warp takes 128 rows of a column:
// a lane joins four consecutive rows (one 32-bit load per residue plane), and
// the results cross shared memory so that C is read and written coalesced.
__global__ void __launch_bounds__(256) crt_join(const unsigned char* __restrict__ res, int slices, int M, int N,
                                                int m_pad, bool upper, Moduli mods, const int* __restrict__ ea,
                                                const int* __restrict__ eb, double2 alpha, double2 beta, double2* C,
                                                long long ldc, double2* C2, int split_col) {
  __shared__ double2 tile[8][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rblocks = m_pad / 128;
  const long long w = blockIdx.x * 8ll + warp;
  const int col = int(w / rblocks), r0 = int(w - (long long)col * rblocks) * 128;
  if (col >= N || (upper && r0 > col)) return;   // wholly below the diagonal: perhaps not computed
  // x / P = frac(sum r f), f = y / p in 32-bit digits f2 f1 f0: below 2^44 per slice in a64, b64
  unsigned c32[8] = {};
  unsigned long long b64[8] = {}, a64[8] = {};
  const unsigned char* src = res + (long long)col * m_pad + r0 + 4 * lane;
  const long long plane = (long long)N * m_pad;
  for (int s = 0; s < slices; ++s) {
#pragma unroll 4
    for (int i = 0; i < kMods; ++i) {
      const unsigned f2 = unsigned(mods.m[i].fhi >> 32), f1 = unsigned(mods.m[i].fhi), f0 = mods.m[i].flo;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const unsigned v = *reinterpret_cast<const unsigned*>(src);
        src += plane;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const unsigned r = (v >> (8 * j)) & 255u;
          c32[2 * j + q] += r * f2;                         // modulo 2^32 above the digit
          b64[2 * j + q] += (unsigned long long)r * f1;
          a64[2 * j + q] += (unsigned long long)r * f0;
        }
      }
    }
  }
  const int e1 = eb[col];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = r0 + 4 * lane + j, e0 = row < M ? ea[row] : 0;
    double v[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const unsigned long long f = ((unsigned long long)c32[2 * j + q] << 32) + b64[2 * j + q] + (a64[2 * j + q] >> 32);
      // centred: |x| < P / 2; the low digit keeps small sums at full precision
      const double s = fma(double(unsigned(a64[2 * j + q])), 0x1p-32, double((long long)f));
      v[q] = fma(s, mods.phi, s * mods.plo);
      v[q] = e0 == kNaN || e1 == kNaN ? nan("") : scalbn(v[q], -(e0 + e1));
    }
    tile[warp][4 * lane + j] = make_double2(v[0], v[1]);
  }
  __syncwarp();
  double2* const out = col < split_col ? C + (long long)col * ldc : C2 + (long long)(col - split_col) * ldc;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = r0 + lane + 32 * j;
    if (row >= M || (upper && row > col)) continue;
    const double2 x = tile[warp][lane + 32 * j];
    double2 o = make_double2(alpha.x * x.x - alpha.y * x.y, alpha.x * x.y + alpha.y * x.x);
    if (beta.x != 0.0 || beta.y != 0.0) {
      const double2 old = out[row];
      o.x += beta.x * old.x - beta.y * old.y;
      o.y += beta.x * old.y + beta.y * old.x;
    }
    out[row] = o;
  }
}

int pad_to(int x, int a) { return (x + a - 1) / a * a; }

// Slices of K: the count with the least estimated time of the tiles' waves
// (about 1 us per step of 128 k and 4 us per CTA) and the longer join.
int pick_slices(int sms, long long tiles, int steps, double mn) {
  int best = 1;
  double best_t = 0;
  for (int s = 1; s <= std::min(8, steps); ++s) {
    const int per = (steps + s - 1) / s, used = (steps + per - 1) / per;
    const double waves = double((tiles * used + sms - 1) / sms);
    const double tm = waves * (per * 1.0e-6 + 4e-6) + used * mn * 2 * kMods / 2.0e12;
    if (best_t == 0 || tm < best_t) {
      best_t = tm;
      best = used;
    }
  }
  return best;
}

constexpr double kMaxBytes = 8e9;   // planes of one operand, and residues of one product

}  // namespace

bool zcrt_serves(int sms, int m, int n, int k, bool a_kept) {
  if (m < 1 || n < 1 || k < 1 || k > kMaxK) return false;
  const double M = m, N = n, K = k;
  const long long tiles = (long long)ceil_div(m, kBM) * ceil_div(n, kBN) * kMods;
  const int steps = ceil_div(k, kKB), s = pick_slices(sms, tiles, steps, M * N), per = ceil_div(steps, s);
  if (double(std::max(crt_plane_bytes(m, k, false), crt_plane_bytes(n, k, true))) > kMaxBytes ||
      double(crt_result_bytes(sms, m, n, k)) > kMaxBytes)
    return false;
  const double native = 8.0 * M * N * K / 36.0e12;
  const double waves = std::ceil(double(tiles) * s / sms);
  const double crt = 40e-6 + ((a_kept ? 0.0 : M) + N) * K * (2 * 16 + 2 * kMods) / 4.0e12 +
                     waves * (per * 1.0e-6 + 4e-6) + M * N * (4.0 * kMods * s + 16) / 3.0e12;
  return crt < 0.85 * native;
}

size_t crt_plane_bytes(int rows, int k, bool as_b) {
  return size_t(2 * kMods) * pad_to(rows, as_b ? kBN : kBM) * pad_to(k, kKB) + size_t(rows) * sizeof(int);
}

size_t crt_result_bytes(int sms, int m, int n, int k) {
  const int mt = ceil_div(m, kBM), nt = ceil_div(n, kBN), steps = ceil_div(k, kKB);
  return size_t(2 * kMods) * pick_slices(sms, (long long)mt * nt * kMods, steps, double(m) * n) * n * mt * kBM;
}

bool crt_reserve(Runtime& rt, size_t a, size_t b, size_t result) {
  return rt.crt_a.try_reserve(a) && rt.crt_b.try_reserve(b) && rt.crt_res.try_reserve(result);
}

CrtPlanes crt_prepare(Runtime& rt, const CrtSide& s, bool as_b, DeviceBuffer<unsigned char>& store) {
  cudaStream_t st = rt.stream;
  CrtPlanes o;
  o.rows = s.rows;
  o.rows_pad = pad_to(s.rows, as_b ? kBN : kBM);
  o.k = s.k;
  o.k_pad = pad_to(s.k, kKB);
  const size_t bytes = size_t(2 * kMods) * o.rows_pad * o.k_pad, need = crt_plane_bytes(s.rows, s.k, as_b);
  if (store.size() < need) store.resize(need);
  unsigned char* planes = store.get();
  int* e = reinterpret_cast<int*>(planes + bytes);   // bytes is a multiple of 1,024
  if (s.kcontig) crt_norm_k<<<s.rows, 256, 0, st>>>(s, e);
  else crt_norm_mn<<<ceil_div(s.rows, 64), 256, 0, st>>>(s, e);
  HALF_LAUNCH("CRT row scales");
  const int blocks = ceil_div((long long)(o.rows_pad / 8) * (o.k_pad / 16), 8);
  if (s.kcontig) crt_split<true><<<blocks, 256, 0, st>>>(s, e, moduli(), o.rows_pad, o.k_pad, planes);
  else crt_split<false><<<blocks, 256, 0, st>>>(s, e, moduli(), o.rows_pad, o.k_pad, planes);
  HALF_LAUNCH("CRT residues");
  rt.prof.launches += 2;
  o.planes = planes;
  o.e = e;
  return o;
}

void crt_product(Runtime& rt, const CrtPlanes& a, const CrtPlanes& b, double2 alpha, double2 beta, double2* C,
                 long long ldc, bool upper, double2* C2, int split_col) {
  cudaStream_t st = rt.stream;
  if (rt.tc_err.size() == 0) {
    rt.tc_err.resize(1);
    rt.tc_err.zero(st);
  }
  const int m = a.rows, n = b.rows, mt = a.rows_pad / kBM, nt = b.rows_pad / kBN, m_pad = a.rows_pad;
  if (a.k != b.k || a.k > kMaxK) fail(kInternal, "CRT product operands do not match");
  const int steps = a.k_pad / kKB;
  const int s = pick_slices(rt.sms, (long long)mt * nt * kMods, steps, double(m) * n), per = ceil_div(steps, s);
  const int slices = ceil_div(steps, per);
  const size_t bytes = crt_result_bytes(rt.sms, m, n, a.k);
  if (rt.crt_res.size() < bytes) rt.crt_res.resize(bytes);
  raise_smem_limit(crt_gemm_kernel, kSmem);
  crt_gemm_kernel<<<dim3(mt, nt, kMods * slices), kThreads, kSmem, st>>>(
      a.planes, b.planes, a.rows_pad, b.rows_pad, a.k_pad, per, n, m_pad, upper, moduli(), rt.crt_res.get(),
      rt.tc_err.get());
  HALF_LAUNCH("CRT product");
  crt_join<<<ceil_div((long long)mt * n, 8), 256, 0, st>>>(
      rt.crt_res.get(), slices, m, n, m_pad, upper, moduli(), a.e, b.e, alpha, beta, C, ldc, C2, split_col);
  HALF_LAUNCH("CRT join");
  rt.prof.launches += 2;
  rt.crt_pending = true;
}

}  // namespace hb
