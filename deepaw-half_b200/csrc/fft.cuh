// Shared-memory mixed-radix FFT engine for pencils of length n <= kMaxFFT,
// used by every transform in the library.
//
// A transform is one, two or (75, 125, 128) three passes over its
// pencils, each pass a register transform of radix 2 .. 12 per thread: the
// kernels that use it are bound by instruction issue and shared-memory
// accesses, and a pass costs one load, one store and one twiddle load per
// point whatever its radix, so few wide passes (96 = 8 x 12) beat many narrow
// ones (96 = 4 x 4 x 2 x 3, up to radix 5; hs.cu has the measured times).  Two in-place orders are provided and chosen per transform so that
// no explicit permutation pass is ever needed:
//   * DIF  (decimation in frequency): natural-order input, output X[k] left at
//     position pos(k) (mixed-radix digit reversal);
//   * DIT  (decimation in time, the transposed algorithm): input x[k] placed
//     at pos(k), natural-order output.
// The scatter into (and the gather out of) the transform is where the
// permutation is absorbed.  fft_pass takes its loads and stores as functors,
// so a kernel can feed the first pass from global memory, skip slots that
// are known to be zero, and store the last pass straight to global memory.
// Sign convention: SIGN = -1 is exp(-2 pi i jk/n) (the reference's FORWARD),
// SIGN = +1 is the unnormalised inverse (CUFFT_INVERSE).
#pragma once

#include <vector>

#include "common.h"

namespace hb {

constexpr int kMaxFFT = 128;
constexpr int kMaxStages = 4;

struct FFTPlan {
  int n = 0;
  int nstages = 0;
  int radix[kMaxStages] = {};
  int span[kMaxStages] = {};   // block length entering stage s (DIF order)
};

inline bool fft_size_supported(int n) {
  if (n < 1 || n > kMaxFFT) return false;
  for (int p : {2, 3, 5})
    while (n % p == 0) n /= p;
  return n == 1;
}

// Fewest passes with register radices, the narrowest widest radix among
// those, radices ascending (the first pass of a DIF transform, which the
// x-line kernel fuses with its potential, gets the narrower one).
inline FFTPlan make_fft_plan(int n) {
  if (!fft_size_supported(n))
    fail(kUnavailable, "FFT grid dimension " + std::to_string(n) + " is not a 2^a 3^b 5^c size up to " +
                           std::to_string(kMaxFFT));
  static const int kRadices[] = {2, 3, 4, 5, 6, 8, 9, 10, 12};   // 16 would need 128 registers in FP64
  FFTPlan p;
  p.n = n;
  std::vector<int> best;
  if (n == 1) {
    best = {1};
  } else {
    for (int r : kRadices)
      if (r == n && r <= 10) best = {r};   // one pass up to 10 points; above, two passes need far fewer registers
    if (best.empty())
      for (int a : kRadices)
        for (int b : kRadices)
          if (a <= b && a * b == n && (best.empty() || b < best.back())) best = {a, b};
    if (best.empty())
      for (int a : kRadices)
        for (int b : kRadices)
          for (int c : kRadices)
            if (a <= b && b <= c && a * b * c == n && (best.empty() || c < best.back())) best = {a, b, c};
    if (best.empty()) fail(kInternal, "no FFT plan for " + std::to_string(n));
  }
  int L = n;
  for (int r : best) {
    p.radix[p.nstages] = r;
    p.span[p.nstages++] = L;
    L /= r;
  }
  return p;
}

// pos[k]: storage position of X[k] after a DIF transform (= input slot of x[k] for DIT)
inline std::vector<int> fft_positions(const FFTPlan& p) {
  std::vector<int> pos(p.n);
  for (int k = 0; k < p.n; ++k) {
    int kk = k, q = 0;
    for (int s = 0; s < p.nstages; ++s) {
      int r = p.radix[s];
      q += (kk % r) * (p.span[s] / r);
      kk /= r;
    }
    pos[k] = q;
  }
  return pos;
}

#ifdef __CUDACC__

template <int SIGN, typename C>
__device__ __forceinline__ C mul_i(C a) {  // (SIGN * i) * a
  C r;
  if (SIGN > 0) { r.x = -a.y; r.y = a.x; }
  else { r.x = a.y; r.y = -a.x; }
  return r;
}

// exp(SIGN 2 pi i K / N) * a with the constant folded in; N = 8 or 9.
template <int N, int K, int SIGN, typename C, typename R>
__device__ __forceinline__ C mul_root(C a) {
  constexpr int k = K % N;
  if (k == 0) return a;
  if (4 * k == N) return mul_i<SIGN, C>(a);
  constexpr double c8[8] = {1, 0.70710678118654752, 0, -0.70710678118654752, -1, -0.70710678118654752, 0,
                            0.70710678118654752};
  constexpr double s8[8] = {0, 0.70710678118654752, 1, 0.70710678118654752, 0, -0.70710678118654752, -1,
                            -0.70710678118654752};
  constexpr double c9[9] = {1, 0.76604444311897804, 0.17364817766693035, -0.5, -0.93969262078590838,
                            -0.93969262078590838, -0.5, 0.17364817766693035, 0.76604444311897804};
  constexpr double s9[9] = {0, 0.64278760968653933, 0.98480775301220806, 0.86602540378443865, 0.34202014332566873,
                            -0.34202014332566873, -0.86602540378443865, -0.98480775301220806, -0.64278760968653933};
  constexpr double cd = N == 8 ? c8[k % 8] : c9[k % 9];
  constexpr double sd = N == 8 ? s8[k % 8] : s9[k % 9];
  constexpr R c = R(cd), s = R(SIGN * sd);
  C r;
  r.x = a.x * c - a.y * s;
  r.y = a.x * s + a.y * c;
  return r;
}

// Register transform y_p = sum_q x_q exp(SIGN 2 pi i p q / N), natural order
// in and out, in place on x[0..N-1].  6, 10 and 12 split into coprime factors
// without twiddles (Good-Thomas), 8 and 9 by Cooley-Tukey.
template <int N, int SIGN, typename C, typename R>
struct RegFFT;

template <int SIGN, typename C, typename R>
struct RegFFT<1, SIGN, C, R> {
  static __device__ __forceinline__ void run(C*) {}
};
template <int SIGN, typename C, typename R>
struct RegFFT<2, SIGN, C, R> {
  static __device__ __forceinline__ void run(C* x) {
    C a = x[0];
    x[0] = cadd(a, x[1]);
    x[1] = csub(a, x[1]);
  }
};
template <int SIGN, typename C, typename R>
struct RegFFT<3, SIGN, C, R> {
  static __device__ __forceinline__ void run(C* x) {
    const R c3 = R(-0.5), s3 = R(0.86602540378443864676372317075294);
    C t = cadd(x[1], x[2]);
    C u = mul_i<SIGN, C>(cscale(csub(x[1], x[2]), s3));
    C base = cadd(x[0], cscale(t, c3));
    x[0] = cadd(x[0], t);
    x[1] = cadd(base, u);
    x[2] = csub(base, u);
  }
};
template <int SIGN, typename C, typename R>
struct RegFFT<4, SIGN, C, R> {
  static __device__ __forceinline__ void run(C* x) {
    C a = cadd(x[0], x[2]), b = csub(x[0], x[2]), c = cadd(x[1], x[3]), d = mul_i<SIGN, C>(csub(x[1], x[3]));
    x[0] = cadd(a, c);
    x[2] = csub(a, c);
    x[1] = cadd(b, d);
    x[3] = csub(b, d);
  }
};
template <int SIGN, typename C, typename R>
struct RegFFT<5, SIGN, C, R> {
  static __device__ __forceinline__ void run(C* x) {
    const R c1 = R(0.30901699437494742410229341718282), s1 = R(0.95105651629515357211643933337938);
    const R c2 = R(-0.80901699437494742410229341718282), s2 = R(0.58778525229247312916870595463907);
    C t1 = cadd(x[1], x[4]), t2 = cadd(x[2], x[3]);
    C u1 = csub(x[1], x[4]), u2 = csub(x[2], x[3]);
    C a1 = cadd(x[0], cadd(cscale(t1, c1), cscale(t2, c2)));
    C a2 = cadd(x[0], cadd(cscale(t1, c2), cscale(t2, c1)));
    C b1 = mul_i<SIGN, C>(cadd(cscale(u1, s1), cscale(u2, s2)));
    C b2 = mul_i<SIGN, C>(csub(cscale(u1, s2), cscale(u2, s1)));
    x[0] = cadd(x[0], cadd(t1, t2));
    x[1] = cadd(a1, b1);
    x[4] = csub(a1, b1);
    x[2] = cadd(a2, b2);
    x[3] = csub(a2, b2);
  }
};

// coprime factors A B: input (B n1 + A n2) mod N, output k at (k mod A, k mod B)
template <int A, int B, int SIGN, typename C, typename R>
__device__ __forceinline__ void reg_fft_coprime(C* x) {
  constexpr int N = A * B;
  C z[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) z[n2][n1] = x[(B * n1 + A * n2) % N];
    RegFFT<A, SIGN, C, R>::run(z[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C y[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) y[n2] = z[n2][k1];
    RegFFT<B, SIGN, C, R>::run(y);
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (k % A == k1) x[k] = y[k % B];
  }
}

// N = A B with twiddles exp(SIGN 2 pi i n2 k1 / N)
template <int A, int B, int SIGN, typename C, typename R, int I = 0>
struct RegTwiddle {
  static __device__ __forceinline__ void run(C (*z)[A]) {
    constexpr int n2 = I / A, k1 = I % A;
    z[n2][k1] = mul_root<A * B, n2 * k1, SIGN, C, R>(z[n2][k1]);
    RegTwiddle<A, B, SIGN, C, R, I + 1>::run(z);
  }
};
template <int A, int B, int SIGN, typename C, typename R>
struct RegTwiddle<A, B, SIGN, C, R, A * B> {
  static __device__ __forceinline__ void run(C (*)[A]) {}
};
template <int A, int B, int SIGN, typename C, typename R>
__device__ __forceinline__ void reg_fft_ct(C* x) {
  C z[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) z[n2][n1] = x[B * n1 + n2];
    RegFFT<A, SIGN, C, R>::run(z[n2]);
  }
  RegTwiddle<A, B, SIGN, C, R>::run(z);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C y[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) y[n2] = z[n2][k1];
    RegFFT<B, SIGN, C, R>::run(y);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = y[k2];
  }
}

#define HB_REG_FFT(N, F, A, B)                                                                  \
  template <int SIGN, typename C, typename R>                                                   \
  struct RegFFT<N, SIGN, C, R> {                                                                \
    static __device__ __forceinline__ void run(C* x) { F<A, B, SIGN, C, R>(x); }                \
  };
HB_REG_FFT(6, reg_fft_coprime, 2, 3)
HB_REG_FFT(10, reg_fft_coprime, 2, 5)
HB_REG_FFT(12, reg_fft_coprime, 3, 4)
HB_REG_FFT(8, reg_fft_ct, 2, 4)
HB_REG_FFT(9, reg_fft_ct, 3, 3)
#undef HB_REG_FFT

// Twiddle table exp(-2 pi i t / n), t < n, filled by the block.
template <typename C>
__device__ __forceinline__ void fill_twiddles(C* tw, int n) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    double s, c;
    sincospi(-2.0 * double(t) / double(n), &s, &c);
    tw[t].x = c;
    tw[t].y = s;
  }
}

// t / d for t, d < 2^16 as a multiply-high: q = floor(t ceil(2^32 / d) / 2^32).
struct FastDiv {
  unsigned d, magic;
  __device__ __forceinline__ explicit FastDiv(int dd)
      : d(unsigned(dd)), magic(dd > 1 ? unsigned(0xFFFFFFFFu / unsigned(dd)) + 1u : 0u) {}
  __device__ __forceinline__ int operator()(int t) const { return d == 1 ? t : int(__umulhi(unsigned(t), magic)); }
};

// One pass of radix RD over npencils pencils: ld(p, i) reads and st(p, i, v)
// writes storage position i of pencil p.  The pencil index runs fastest over
// the threads.  Callers put a barrier between two passes over the same data.
template <int RD, bool DIT, int SIGN, typename C, typename R, typename Ld, typename St>
__device__ __forceinline__ void fft_pass_radix(const FFTPlan& plan, int s, int npencils, const C* tw, Ld ld, St st) {
  const int n = plan.n, L = plan.span[s], m = L / RD, per = n / RD, tunit = n / L;
  const int total = npencils * per;
  const FastDiv by_pencils(npencils), by_m(m);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int b = by_pencils(t), p = t - b * npencils;
    const int blk = L == n ? 0 : by_m(b), j = b - blk * m;
    const int i0 = blk * L + j;
    C x[RD];
#pragma unroll
    for (int q = 0; q < RD; ++q) x[q] = ld(p, i0 + q * m);
    const int tj = j * tunit;
    if (DIT && m > 1) {
#pragma unroll
      for (int q = 1; q < RD; ++q) {
        C w = tw[q * tj];
        if (SIGN > 0) w.y = -w.y;
        x[q] = cmul(x[q], w);
      }
    }
    RegFFT<RD, SIGN, C, R>::run(x);
    if (!DIT && m > 1) {
#pragma unroll
      for (int q = 1; q < RD; ++q) {
        C w = tw[q * tj];
        if (SIGN > 0) w.y = -w.y;
        x[q] = cmul(x[q], w);
      }
    }
#pragma unroll
    for (int q = 0; q < RD; ++q) st(p, i0 + q * m, x[q]);
  }
}

#define HB_FFT_SWITCH(radix, CALL) \
  switch (radix) {                 \
    case 1: CALL(1); break;        \
    case 2: CALL(2); break;        \
    case 3: CALL(3); break;        \
    case 4: CALL(4); break;        \
    case 5: CALL(5); break;        \
    case 6: CALL(6); break;        \
    case 8: CALL(8); break;        \
    case 9: CALL(9); break;        \
    case 10: CALL(10); break;      \
    default: CALL(12); break;      \
  }

template <bool DIT, int SIGN, typename C, typename R, typename Ld, typename St>
__device__ __forceinline__ void fft_pass(const FFTPlan& plan, int s, int npencils, const C* tw, Ld ld, St st) {
#define HB_CALL(RD) fft_pass_radix<RD, DIT, SIGN, C, R>(plan, s, npencils, tw, ld, st)
  HB_FFT_SWITCH(plan.radix[s], HB_CALL)
#undef HB_CALL
}

// The last pass of an inverse DIT transform, mid(p, i, v) on every point in
// natural order, and the first pass of a forward DIF transform: both passes
// own the same points, so they stay in registers in between.
template <int RD, typename C, typename R, typename Ld, typename Mid, typename St>
__device__ __forceinline__ void fft_pass_fused_radix(const FFTPlan& plan, int npencils, const C* tw, Ld ld, Mid mid,
                                                     St st) {
  const int m = plan.n / RD;
  const int total = npencils * m;
  const FastDiv by_pencils(npencils);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int j = by_pencils(t), p = t - j * npencils;
    C x[RD];
#pragma unroll
    for (int q = 0; q < RD; ++q) x[q] = ld(p, j + q * m);
    if (m > 1) {
#pragma unroll
      for (int q = 1; q < RD; ++q) x[q] = cconjmul(tw[q * j], x[q]);
    }
    RegFFT<RD, +1, C, R>::run(x);
#pragma unroll
    for (int q = 0; q < RD; ++q) x[q] = mid(p, j + q * m, x[q]);
    RegFFT<RD, -1, C, R>::run(x);
    if (m > 1) {
#pragma unroll
      for (int q = 1; q < RD; ++q) x[q] = cmul(x[q], tw[q * j]);
    }
#pragma unroll
    for (int q = 0; q < RD; ++q) st(p, j + q * m, x[q]);
  }
}

template <typename C, typename R, typename Ld, typename Mid, typename St>
__device__ __forceinline__ void fft_pass_fused(const FFTPlan& plan, int npencils, const C* tw, Ld ld, Mid mid, St st) {
#define HB_CALL(RD) fft_pass_fused_radix<RD, C, R>(plan, npencils, tw, ld, mid, st)
  HB_FFT_SWITCH(plan.radix[0], HB_CALL)
#undef HB_CALL
}

// In-place forward or inverse DIF transform of `npencils` pencils in shared
// memory; element k of pencil p lives at buf[p * pstride + k * estride].
template <int SIGN, typename C, typename R>
__device__ void fft_pencils(C* buf, int npencils, int pstride, int estride, const FFTPlan& plan, const C* tw) {
  auto ld = [&](int p, int i) { return buf[p * pstride + i * estride]; };
  auto st = [&](int p, int i, C v) { buf[p * pstride + i * estride] = v; };
  for (int s = 0; s < plan.nstages; ++s) {
    fft_pass<false, SIGN, C, R>(plan, s, npencils, tw, ld, st);
    __syncthreads();
  }
}

// Plan + position table as kernel arguments (passed by value).
struct AxisPlan {
  FFTPlan plan;
  int pos[kMaxFFT];
};

inline AxisPlan make_axis_plan(int n) {
  AxisPlan a;
  a.plan = make_fft_plan(n);
  auto p = fft_positions(a.plan);
  for (int k = 0; k < n; ++k) a.pos[k] = p[k];
  for (int k = n; k < kMaxFFT; ++k) a.pos[k] = 0;
  return a;
}

#endif  // __CUDACC__

}  // namespace hb
