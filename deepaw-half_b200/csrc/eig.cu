// Small dense Hermitian eigensolvers for the ACC subspace problems, device
// resident and free of host synchronisation.
//
// The reference calls cuSOLVER zheevd (m x m metric) and zhegvd (2m x 2m
// Rayleigh-Ritz) once per iteration (src/half_cuda_iterative_solver.cuf:
// 242-275).  For the sizes the solver meets (m <= a few hundred) those calls
// are dominated by per-reflector back-transformation launches and a host
// round trip.  Here the same reduction -- X with X^H B X = I, C = X^H A X,
// Householder tridiagonalisation, Y = X V -- runs in kernels that keep the
// matrix in the shared memory of a cluster of CTAs (orders to 432):
//
//   metric_factor_kernel   X = D R^-1 from a Cholesky factorisation, its pivots
//                          floored (metrics, pencils to order 164) or reported;
//   hetrd_kernel           tridiagonalisation (both also over the whole GPU's
//                          shared memory, orders 434 to 1,280, with cuSOLVER's
//                          zunmtr behind them);
//   tridiag_values_kernel  eigenvalues of the real symmetric tridiagonal T by
//                          multisection on Sturm counts (one warp per
//                          eigenvalue, CTAs across the GPU);
//   tridiag_vectors_kernel eigenvectors by inverse iteration on the pivoted
//                          tridiagonal LU (one thread per eigenvector);
//                          eigenvalues closer than 1e-7 ||T|| form clusters
//                          whose members a warp iterates together and
//                          Gram-Schmidt orthogonalises in order (after
//                          LAPACK's dstebz/dstein); above order 164 a step of
//                          Z (3/2 - Z^T Z / 2) makes them orthogonal to rounding;
//   back_transform_kernel  V = Q Z with Q = H(n-1)...H(1), the reflectors
//                          staged in shared memory, one warp per eigenvector.
//
// Y^H B Y = I, the same normalisation as zhegvd (itype 1, upper).
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>

#include <cfloat>
#include <cmath>
#include <string>

#include "blas.h"
#include "blockops.h"
#include "context.h"
#include "eig.h"

namespace hb {

namespace cg = cooperative_groups;

namespace {

constexpr int kExtraEig = 8;   // eigenvalues located beyond the wanted ones (cluster at the cut)
constexpr size_t kSmemMax = 226 * 1024;   // dynamic shared memory per CTA, leaving room for static

// Number of eigenvalues of T below x (Sylvester inertia of T - x I), T scaled
// to a norm of at most 1 with squared off-diagonals floored at kE2Floor.  The
// pivots of the LDL^T factorisation are ratios q_i = p_i / p_{i-1} of the
// continuant p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}, so the count is the
// number of sign changes along p_0 = 1, p_1, ..., p_n.  Carrying p instead of
// q keeps divisions off the dependent chain, which is one FMA per step: the
// sign test works on the high words beside it, and the pair (p_{i-1}, p_i) is
// rescaled by a power of two (which changes no ratio) only every four steps.
// Per step the larger of the pair grows by at most |d - x| + e^2 <= 3 and
// shrinks by at most kE2Floor / 4, so four steps from 2^-300 stay above
// 2^-790.  That also means no pivot needs a floor of its own: a zero p_i is
// followed by -e^2 p_{i-1}, and either sign given to it counts one change.
// (One rescaling branch and a pivot test per step made a step about 170
// cycles; order 144, 80 values: 116 us.)
constexpr double kE2Floor = 0x1p-120;   // moves e by 2^-60 of the norm at most, below eps / 2 of it

__device__ __forceinline__ void sturm_step(double di, double e2, double x, double& p0, double& p1, int& c) {
  const double p2 = fma(di - x, p1, -e2 * p0);
  c += (__double2hiint(p2) ^ __double2hiint(p1)) < 0;
  p0 = p1;
  p1 = p2;
}

__device__ __forceinline__ void sturm_rescale(double& p0, double& p1) {
  const int ex = (__double2hiint(fabs(p0) > fabs(p1) ? p0 : p1) >> 20) & 0x7ff;   // biased exponent of the larger
  if (ex > 1023 + 300 || ex < 1023 - 300) {
    const double sc = __hiloint2double((2046 - max(ex, 1)) << 20, 0);   // 2^-(ex - 1023)
    p0 *= sc;
    p1 *= sc;
  }
}

__device__ int sturm_count(const double* d, const double* e2, int n, double x) {
  double p0 = 1.0, p1 = d[0] - x;
  int c = __double2hiint(p1) < 0;
  int i = 1;
  for (; i + 3 < n; i += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) sturm_step(d[i + q], e2[i + q - 1], x, p0, p1, c);
    sturm_rescale(p0, p1);
  }
  for (; i < n; ++i) sturm_step(d[i], e2[i - 1], x, p0, p1, c);
  return c;
}

// LU factorisation with partial pivoting of T - lambda I (O(n)); the pivots
// are stored inverted so that the solves multiply.  ai, b1, b2, l and piv are
// per-thread scratch of n elements at stride st (the slots of a group of
// threads are interleaved, so a warp touches consecutive words).
__device__ void tri_factor(const double* d, const double* e, int n, double lam, double tiny, double* ai, double* b1,
                           double* b2, double* l, unsigned char* piv, int st) {
  double diag = d[0] - lam, sup = n > 1 ? e[0] : 0.0;
  for (int i = 0; i < n - 1; ++i) {
    const double sub = e[i];
    const double nd = d[i + 1] - lam, ns = (i + 1 < n - 1) ? e[i + 1] : 0.0;
    const int o = i * st;
    if (fabs(diag) >= fabs(sub)) {
      if (fabs(diag) < tiny) diag = diag < 0 ? -tiny : tiny;
      const double r = 1.0 / diag, m = sub * r;
      ai[o] = r; b1[o] = sup; b2[o] = 0.0; l[o] = m; piv[o] = 0;
      diag = nd - m * sup;
      sup = ns;
    } else {
      const double r = 1.0 / sub, m = diag * r;
      ai[o] = r; b1[o] = nd; b2[o] = ns; l[o] = m; piv[o] = 1;
      diag = sup - m * nd;
      sup = -m * ns;
    }
  }
  if (fabs(diag) < tiny) diag = diag < 0 ? -tiny : tiny;
  const int o = (n - 1) * st;
  ai[o] = 1.0 / diag;
  b1[o] = 0.0;
  b2[o] = 0.0;
}

// The running values of both sweeps stay in registers, so the dependent
// chain of a step is one or two FMAs, not a shared-memory round trip.
__device__ void tri_solve(int n, const double* ai, const double* b1, const double* b2, const double* l,
                          const unsigned char* piv, double* x, int st) {
  double cur = x[0];
  for (int i = 0; i < n - 1; ++i) {   // forward: L^-1 with the row swaps
    const int o = i * st;
    const double nxt = x[o + st], li = l[o];
    if (piv[o]) {
      x[o] = nxt;
      cur = cur - li * nxt;
    } else {
      x[o] = cur;
      cur = nxt - li * cur;
    }
  }
  const int on = (n - 1) * st;
  double x1 = cur * ai[on];   // x(i+1)
  x[on] = x1;
  if (n == 1) return;
  const int om = (n - 2) * st;
  double x0 = (x[om] - b1[om] * x1) * ai[om];   // x(i)
  x[om] = x0;
  for (int i = n - 3; i >= 0; --i) {   // backward: U^-1
    const int o = i * st;
    const double xi = (x[o] - b1[o] * x0 - b2[o] * x1) * ai[o];
    x[o] = xi;
    x1 = x0;
    x0 = xi;
  }
}

// Padded Gershgorin interval of T and the norm max_i (|d_i| + |e_{i-1}| + |e_i|),
// by one warp; every lane gets the results.  Both tridiagonal kernels evaluate
// it with this one routine, so they agree bit for bit.
__device__ void gershgorin(const double* d, const double* e, int n, double& lo, double& hi, double& nrm) {
  double gl = d[0], gu = d[0];
  nrm = 0;
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    gl = fmin(gl, d[i] - r);
    gu = fmax(gu, d[i] + r);
    nrm = fmax(nrm, fabs(d[i]) + r);
  }
  for (int off = 16; off > 0; off >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, off));
    gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, off));
    nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, off));
  }
  const double pad = 2.0 * DBL_EPSILON * fmax(fabs(gl), fabs(gu)) * n + 1e-300;
  lo = gl - pad;
  hi = gu + pad;
  nrm = fmax(nrm, DBL_MIN);
}

// Power of two that brings a norm below 1.
__device__ __forceinline__ double norm_scale(double nrm) { return scalbn(1.0, -(ilogb(nrm) + 1)); }

// Squared off-diagonal of the scaled T, floored for sturm_count.
__device__ __forceinline__ double scaled_e2(double e, double sc) { return fmax((e * sc) * (e * sc), kE2Floor); }

constexpr int kValueWarps = 8;       // eigenvalues per CTA of the value kernel, one warp each
constexpr int kVectorThreads = 32;   // eigenvectors per CTA of the vector kernel, one thread each

// Eigenvalue k of the scaled T in [lo, hi] by multisection: the 32 lanes of a
// warp count at 32 interior points of the bracket per round, which shrinks to
// the pair of neighbouring points whose counts straddle the index (33-fold
// per round).  Brackets end at 2 eps |lambda| + eps ||T|| (absolute accuracy
// eps ||T||, as bisection guarantees).
__device__ double multisect(const double* d, const double* e2, int n, int k, double lo, double hi, double tnorm) {
  const int lane = threadIdx.x & 31;
  for (int round = 0; round < 200; ++round) {   // lo and hi are warp-uniform throughout
    if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + DBL_EPSILON * tnorm) break;
    const double x = lo + (hi - lo) * double(lane + 1) / 33.0;
    const unsigned b = __ballot_sync(0xffffffffu, sturm_count(d, e2, n, x) > k);   // lambda_k < x
    const int first = b ? __ffs(b) - 1 : 32;                                          // first point above
    const double xlo = __shfl_sync(0xffffffffu, x, first > 0 ? first - 1 : 0);
    const double xhi = __shfl_sync(0xffffffffu, x, first < 32 ? first : 31);
    const double nlo = first > 0 ? xlo : lo, nhi = first < 32 ? xhi : hi;
    if (!(nlo > lo || nhi < hi)) break;   // no progress left in floating point
    lo = nlo;
    hi = nhi;
  }
  return 0.5 * (lo + hi);
}

// Eigenvalues 0..ne-1 of T (ascending), one warp each.  Also sets *status for
// the vector kernel that follows on the stream: 0, or kWaitGaveUp when a grid
// barrier of the tridiagonalisation gave up.
__global__ void __launch_bounds__(32 * kValueWarps) tridiag_values_kernel(const double* __restrict__ d_in,
                                                                          const double* __restrict__ e_in, int n,
                                                                          int ne, double* __restrict__ lam,
                                                                          const int* __restrict__ grid_err,
                                                                          int* __restrict__ status) {
  wait_previous();
  extern __shared__ double sm[];
  double* d = sm;
  double* e = d + n;
  double* e2 = e + n;
  __shared__ double s_gl, s_gu, s_norm;
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = grid_err && *grid_err ? kWaitGaveUp : 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] = d_in[i];
    e[i] = i < n - 1 ? e_in[i] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double gl, gu, nrm;
    gershgorin(d, e, n, gl, gu, nrm);
    if (threadIdx.x == 0) { s_gl = gl; s_gu = gu; s_norm = nrm; }
  }
  __syncthreads();
  const double sc = norm_scale(s_norm);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] *= sc;
    e2[i] = scaled_e2(e[i], sc);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * kValueWarps + (threadIdx.x >> 5);
  if (k >= ne) return;   // whole warps; no barrier follows
  const double v = multisect(d, e2, n, k, s_gl * sc, s_gu * sc, s_norm * sc);
  if (lane == 0) lam[k] = v / sc;
}

// x(i) of a slot, scaled to norm 1; the norm before.
__device__ double normalise(double* x, int n, int st) {
  double nrm = 0;
  for (int i = 0; i < n; ++i) nrm += x[i * st] * x[i * st];
  nrm = sqrt(nrm);
  const double inv = 1.0 / nrm;
  for (int i = 0; i < n; ++i) x[i * st] *= inv;
  return nrm;
}

// The same and Gram-Schmidt by the whole warp: lane = slot + per q, and the
// 32 / per lanes of a slot share its vector (elements q, q + 32 / per, ...).
__device__ __forceinline__ double slot_sum(double v, int per) {
  for (int off = per; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__device__ double slot_normalise(double* x, int n, int st, int per, bool on) {
  const int q = (threadIdx.x & 31) / per, g = 32 / per;
  double s = 0;
  for (int i = q; i < n; i += g) s += x[i * st] * x[i * st];
  const double nrm = sqrt(slot_sum(s, per));
  if (on) {
    const double inv = 1.0 / nrm;
    for (int i = q; i < n; i += g) x[i * st] *= inv;
  }
  return nrm;
}

// x -= sum_j (y_j . x) y_j over NY vectors, stride sy and one after another at distance dy.
template <int NY>
__device__ void slot_remove(double* x, int st, const double* y, int sy, size_t dy, int n, int per, bool on) {
  const int q = (threadIdx.x & 31) / per, g = 32 / per;
  double s[NY] = {};
#pragma unroll 8
  for (int i = q; i < n; i += g) {
    const double v = x[i * st];
#pragma unroll
    for (int j = 0; j < NY; ++j) s[j] += y[j * dy + size_t(i) * sy] * v;
  }
#pragma unroll
  for (int j = 0; j < NY; ++j) s[j] = slot_sum(s[j], per);   // every lane takes part
  if (!on) return;
#pragma unroll 8
  for (int i = q; i < n; i += g) {
    double v = x[i * st];
#pragma unroll
    for (int j = 0; j < NY; ++j) v -= s[j] * y[j * dy + size_t(i) * sy];
    x[i * st] = v;
  }
}

// z = x with its largest component positive.
__device__ void store_signed(double* __restrict__ z, const double* x, int n, int st) {
  double big = 0;
  for (int i = 0; i < n; ++i)
    if (fabs(x[i * st]) > fabs(big)) big = x[i * st];
  const double sg = big < 0 ? -1.0 : 1.0;
  for (int i = 0; i < n; ++i) z[i] = sg * x[i * st];
}

// Start vector of eigenvector k, deterministic and pseudo-random; of either
// sign in a cluster, whose members differ by it.
__device__ void start_vector(double* x, int n, int st, int k, bool clustered) {
  unsigned s = 0x9E3779B9u * (k + 1);
  for (int i = 0; i < n; ++i) {
    s = s * 1664525u + 1013904223u;
    const double u = double(s >> 8) / 16777216.0 - 0.5;
    x[i * st] = clustered ? u : 1.0 + 0.5 * u;
  }
}

// tridiag_vectors_kernel's work on the cnt values from c0 on when some of them
// are members of clusters; true when the lane's vector is in order.  A call, so
// that the kernel's path without clusters keeps its registers.
__device__ __noinline__ bool cluster_batch(const double* d, const double* e, const double* lam, const int* cl_first,
                                           int n, int per, int c0, int cnt, bool clustered, double tiny, double tnorm,
                                           double* ai, double* b1, double* b2, double* l, double* x,
                                           unsigned char* piv, int st, const double* Z) {
  const int lane = threadIdx.x, k = c0 + lane, slot = min(lane, per - 1);
  const bool on = lane < cnt;
  const int f = on ? cl_first[k] : 0;                               // first member
  const int base = max(f, c0) - c0, pos = on ? lane - base : 0;     // of the batch's members: lane of the first, place
  int steps = on ? 1 : 0;                                           // members in the batch
  while (on && base + steps < cnt && cl_first[c0 + base + steps] == f) ++steps;
  for (int off = 16; off > 0; off >>= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, off));
  // the Gram-Schmidt's view: lane = gs + per q works on slot gs, its vector, cluster and place
  const int gs = lane & (per - 1);
  double* const gx = x + (gs - slot);
  const int gf = __shfl_sync(0xffffffffu, f, gs), gbase = __shfl_sync(0xffffffffu, base, gs);
  const int gpos = __shfl_sync(0xffffffffu, pos, gs);
  const bool gclustered = __shfl_sync(0xffffffffu, int(clustered), gs);
  if (on) {
    double lk = lam[f];
    for (int q = f + 1; q <= k; ++q) {   // numerically equal eigenvalues of a cluster are separated (dstein)
      const double sep = 10.0 * DBL_EPSILON * fmax(fabs(lam[q]), tnorm * 1e-3);
      lk = lam[q] - lk < sep ? lk + sep : lam[q];
    }
    tri_factor(d, e, n, lk, tiny, ai, b1, b2, l, piv, st);
    start_vector(x, n, st, k, clustered);
  }
  bool ok = true;
  for (int it = 0; it < 3; ++it) {
    if (on && (clustered || it < 2)) {
      tri_solve(n, ai, b1, b2, l, piv, x, st);
      const double nrm = normalise(x, n, st);
      ok = ok && nrm > 0 && isfinite(nrm);
    }
    for (int pass = 0; pass < (it == 2 ? 2 : 1); ++pass) {
      __syncwarp();
      int j = cl_first[c0];   // only the batch's first cluster can have members that are done
      const bool part = gclustered && gf < c0;
      if (it == 0) j = c0;    // and from the second round on: the first leaves the vectors different enough
      // four at a time: as many as the L1 beside the scratch holds for the second reading
      for (; j + 3 < c0; j += 4) slot_remove<4>(gx, st, Z + (size_t)j * n, 1, n, n, per, part);
      for (; j < c0; ++j) slot_remove<1>(gx, st, Z + (size_t)j * n, 1, n, n, per, part);
      __syncwarp();
      for (int r = 0; r < steps; ++r) {
        const double nrm = slot_normalise(gx, n, st, per, gclustered && gpos == r);
        if (gclustered && gpos == r) ok = ok && nrm > 0 && isfinite(nrm);
        __syncwarp();
        slot_remove<1>(gx, st, gx + (min(gbase + r, per - 1) - gs), st, 0, n, per, gclustered && gpos > r);
        __syncwarp();
      }
    }
  }
  return ok;
}

// Eigenvectors of lam[0..nev) by inverse iteration on the pivoted LU of
// T - lambda I, one thread per eigenvector.  Eigenvalues (up to ne) closer
// than 1e-7 ||T|| form clusters, whose members are orthogonalised against each
// other (LAPACK's dstein does the same with 1e-3 ||T||, which would take most
// of the dense Ritz spectra met here).  Outside a cluster inverse iteration
// alone keeps |<z_i, z_j>| <= eps ||T|| / gap <~ 1e-9.
//
// A cluster belongs to the CTA (one warp) of its first member.  The warp takes
// `per` consecutive values at a time, a lane each: all solve, then modified
// Gram-Schmidt inside each cluster, in ascending order, against the members
// that are done (in Z) and those of the batch, all 32 lanes working on the
// batch's vectors.  Three such rounds, the last one with a second pass.  With
// one thread for a whole cluster, the solves of the undisplaced 64-atom cell at
// (1/2, 1/2, 1/2), whose levels are many-fold, took 299 and 740 ms with 160 and
// 400 bands; like this 109 and 246 ms (with cuSOLVER's pencils 138 and 305).
//
// Scratch: five n-vectors and the pivot flags per thread, interleaved by thread
// (a warp touches consecutive words), in shared memory after the tables when
// gscratch is null, else in global memory with one slot per eigenvector.  A CTA takes `per` eigenvectors,
// as many as its shared memory holds (32 at order 138, 8 at order 432): the
// threads run serial chains, so few of them per SM cost nothing, while
// scratch in global memory puts a cache miss into every link.
__global__ void __launch_bounds__(kVectorThreads) tridiag_vectors_kernel(
    const double* __restrict__ d_in, const double* __restrict__ e_in, int n, int nev, int ne, int per,
    const double* __restrict__ lam_g, double* __restrict__ w, double* Z, double* __restrict__ gscratch,
    int* __restrict__ status, const int* __restrict__ failed) {
  wait_previous();
  const int stop = failed ? *failed : 0;
  extern __shared__ double sm[];
  double* d = sm;
  double* e = d + n;
  double* lam = e + n;
  int* cl_first = reinterpret_cast<int*>(lam + ne);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] = d_in[i];
    e[i] = i < n - 1 ? e_in[i] : 0.0;
  }
  for (int i = threadIdx.x; i < ne; i += blockDim.x) lam[i] = lam_g[i];
  if (stop) return;
  __syncthreads();
  double gl, gu, tnorm;   // one warp (kVectorThreads) evaluates, every thread holds the results
  gershgorin(d, e, n, gl, gu, tnorm);
  const double ortol = 1.0e-7 * tnorm;
  for (int k = threadIdx.x; k < ne; k += blockDim.x) {   // first member of each value's cluster
    int f = k;
    while (f > 0 && !(lam[f] - lam[f - 1] > ortol)) --f;
    cl_first[k] = f;
  }
  __syncthreads();
  const int lane = threadIdx.x, slot = min(lane, per - 1);
  const double tiny = DBL_EPSILON * tnorm;
  double* ai;
  unsigned char* piv;
  int st;
  if (gscratch) {
    st = gridDim.x * per;
    ai = gscratch + blockIdx.x * per + slot;
    piv = reinterpret_cast<unsigned char*>(gscratch + 5 * size_t(n) * st) + blockIdx.x * per + slot;
  } else {
    size_t off = (2 * size_t(n) + ne) * sizeof(double) + size_t(ne) * sizeof(int);
    off = (off + 15) & ~size_t(15);
    double* sbase = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(sm) + off);
    st = per;
    ai = sbase + slot;
    piv = reinterpret_cast<unsigned char*>(sbase + 5 * size_t(n) * st) + slot;
  }
  double* b1 = ai + size_t(n) * st;
  double* b2 = b1 + size_t(n) * st;
  double* l = b2 + size_t(n) * st;
  double* x = l + size_t(n) * st;
  if (lane < per && blockIdx.x * per + lane < nev) w[blockIdx.x * per + lane] = lam[blockIdx.x * per + lane];
  // this CTA's values: the clusters that begin among its `per`, whole
  auto cluster_start = [&](int k) {
    while (k < ne && cl_first[k] != k) ++k;
    return k;
  };
  const int kbeg = cluster_start(blockIdx.x * per);
  const int kend = kbeg < nev ? cluster_start(min((int(blockIdx.x) + 1) * per, nev)) : kbeg;
  for (int c0 = kbeg; c0 < kend; c0 += per) {
    const int cnt = min(per, kend - c0), k = c0 + lane;
    const bool on = lane < cnt;
    const bool clustered = on && (cl_first[k] < k || (k + 1 < ne && cl_first[k + 1] == k));
    bool ok = true;
    if (__any_sync(0xffffffffu, clustered)) {
      ok = cluster_batch(d, e, lam, cl_first, n, per, c0, cnt, clustered, tiny, tnorm, ai, b1, b2, l, x, piv, st, Z);
    } else if (on) {
      tri_factor(d, e, n, lam[k], tiny, ai, b1, b2, l, piv, st);
      start_vector(x, n, st, k, false);
      // With an eigenvalue accurate to rounding each solve amplifies the wanted
      // direction by ~gap / (eps ||T||): two are enough.
      for (int it = 0; it < 2; ++it) {
        tri_solve(n, ai, b1, b2, l, piv, x, st);
        const double nrm = normalise(x, n, st);
        ok = ok && nrm > 0 && isfinite(nrm);
      }
    }
    if (!__all_sync(0xffffffffu, ok)) {   // the rest is of no use either
      if (lane == 0) atomicCAS(status, 0, 1);   // an earlier report stays
      return;
    }
    if (on) store_signed(Z + (size_t)k * n, x, n, st);
    __syncwarp();
  }
}

constexpr int kBackWarps = 4;      // eigenvectors per CTA of the back-transformation, one warp each
constexpr int kBackBlock = 4;      // reflectors applied together

__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// Sums over the warp of eight values per lane at once: afterwards `v[0]` of
// lane l holds the sum of value l >> 2 (9 exchanges instead of 40).
__device__ __forceinline__ double warp_sum8(double (&v)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 4, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// V[:, j] = Q z_j with Q = H(n-1) ... H(1) (LAPACK zhetrd, UPLO = 'U':
// v(i) = 1, v(1:i-1) = A(1:i-1, i+1), tau(i)).  One warp per eigenvector, the
// vector in registers (row lane + 32 t in slot t < RX); the CTA's warps share
// the reflectors, staged in shared memory `chunk` at a time (v with its unit
// entry and zeros below).  A reflector by itself is a dot product, a
// five-step shuffle reduction and an update, all dependent; four at a time
// share one reduction: with d_i = v_i^H x and the Gram g_ij = v_i^H v_j
// (j < i),  w_i = tau_i (d_i - sum_j g_ij w_j)  and  x -= sum_i w_i v_i.
template <int RX>
__global__ void __launch_bounds__(32 * kBackWarps) back_transform_kernel(const double2* __restrict__ A,
                                                                         const double2* __restrict__ tau,
                                                                         const double* __restrict__ Z, int n, int nev,
                                                                         int chunk, double2* __restrict__ V) {
  wait_previous();
  extern __shared__ __align__(16) double2 vs[];     // chunk x n
  double2* ts = vs + (size_t)chunk * n;             // chunk
  double2* gram = ts + chunk;                       // chunk / 4 x 8: g10, g20, g21, g30, g31, g32
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * kBackWarps + warp;
  const bool active = j < nev;
  double2 x[RX];
#pragma unroll
  for (int t = 0; t < RX; ++t) {
    const int r = lane + 32 * t;
    x[t] = make_double2(active && r < n ? Z[(size_t)j * n + r] : 0.0, 0.0);
  }
  for (int c0 = 0; c0 <= n - 2; c0 += chunk) {
    const int cnt = min(chunk, n - 1 - c0);
    const int blocks = (cnt + kBackBlock - 1) / kBackBlock;
    __syncthreads();   // the previous chunk is consumed
    for (int q = warp; q < blocks * kBackBlock; q += kBackWarps) {   // reflectors beyond the last: zero
      const int i0 = c0 + q;
      for (int r = lane; r < n; r += 32) {
        if (q < cnt && r < i0) copy16_async(vs + (size_t)q * n + r, A + (size_t)(i0 + 1) * n + r);
        else vs[(size_t)q * n + r] = make_double2(q < cnt && r == i0 ? 1.0 : 0.0, 0.0);
      }
      if (lane == 0) ts[q] = q < cnt ? tau[i0] : make_double2(0.0, 0.0);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int b = warp; b < blocks; b += kBackWarps) {
      const double2* v0 = vs + (size_t)b * kBackBlock * n;
      double g[2][8] = {};
      for (int r = lane; r < min(n, c0 + (b + 1) * kBackBlock); r += 32) {
        const double2 a0 = v0[r], a1 = v0[n + r], a2 = v0[2 * n + r], a3 = v0[3 * n + r];
        auto dot = [](double* o, double2 p, double2 q) {   // conj(p) q
          o[0] += p.x * q.x + p.y * q.y;
          o[1] += p.x * q.y - p.y * q.x;
        };
        dot(g[0], a1, a0);
        dot(g[0] + 2, a2, a0);
        dot(g[0] + 4, a2, a1);
        dot(g[0] + 6, a3, a0);
        dot(g[1], a3, a1);
        dot(g[1] + 2, a3, a2);
      }
      double* out = reinterpret_cast<double*>(gram + b * 8);
      const double s0 = warp_sum8(g[0]), s1 = warp_sum8(g[1]);
      if ((lane & 3) == 0) {
        out[lane >> 2] = s0;
        if ((lane >> 2) < 4) out[8 + (lane >> 2)] = s1;
      }
    }
    __syncthreads();
    if (!active) continue;
    for (int b = 0; b < blocks; ++b) {
      const double2* v = vs + (size_t)b * kBackBlock * n;
      const int rows = min(n, c0 + (b + 1) * kBackBlock);   // rows 0 .. i0 of the block's last reflector
      double d[8] = {};
#pragma unroll
      for (int t = 0; t < RX; ++t) {
        const int r = lane + 32 * t;
        if (r < rows) {
#pragma unroll
          for (int i = 0; i < kBackBlock; ++i) {
            const double2 a = v[i * n + r];
            d[2 * i] += a.x * x[t].x + a.y * x[t].y;
            d[2 * i + 1] += a.x * x[t].y - a.y * x[t].x;
          }
        }
      }
      const double mine = warp_sum8(d);
      double2 w[kBackBlock];
#pragma unroll
      for (int i = 0; i < kBackBlock; ++i) {
        w[i].x = __shfl_sync(0xffffffffu, mine, 8 * i);
        w[i].y = __shfl_sync(0xffffffffu, mine, 8 * i + 4);
      }
      const double2* g = gram + b * 8;
#pragma unroll
      for (int i = 0; i < kBackBlock; ++i) {
#pragma unroll
        for (int k = 0; k < i; ++k) w[i] = csub(w[i], cmul(g[i * (i - 1) / 2 + k], w[k]));
        w[i] = cmul(ts[b * kBackBlock + i], w[i]);
      }
#pragma unroll
      for (int t = 0; t < RX; ++t) {
        const int r = lane + 32 * t;
        if (r < rows) {
#pragma unroll
          for (int i = 0; i < kBackBlock; ++i) x[t] = csub(x[t], cmul(v[i * n + r], w[i]));
        }
      }
    }
  }
  if (active) {
#pragma unroll
    for (int t = 0; t < RX; ++t) {
      const int r = lane + 32 * t;
      if (r < n) V[(size_t)j * n + r] = x[t];
    }
  }
}

// lower triangle from the upper one (Hermitian)
__global__ void hermitian_fill_kernel(double2* A, int n) {
  after_previous();
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)n * n) return;
  int j = int(t / n), i = int(t - (long long)j * n);
  if (i > j) {
    double2 u = A[(long long)i * n + j];
    A[t] = make_double2(u.x, -u.y);
  } else if (i == j) {
    A[t].y = 0.0;
  }
}

// S-metric normalisation of the ACC correction block without an
// eigendecomposition.  Given M = P^H S P (m x m, upper triangle read), write
// U (m x m, upper triangular) with (P U)^H S (P U) = I up to the floor:
//   D = diag(M)^-1/2,  D M D = R^H R (Cholesky, pivots floored at 1e-14),
//   U = D R^-1.
// P U spans what P spans (the reference's eigenvector basis U Lambda^-1/2
// spans the same space), so the Rayleigh-Ritz step that follows sees the
// same subspace; the floor plays the role of the reference's 1e-14 floor on
// the metric eigenvalues for nearly dependent directions: a pivot at or below
// 1e-14 (of the unit scaled diagonal) gives R(k,k) = 1e-7 and a zero row, so
// the direction stays in the span without being eliminated from later
// columns.
//
// One right-looking sweep builds R^-1 together with R.  With
// T(i,j) = sum_{l<j} X(i,l) R(l,j) for i < j (X = R^-1), step k is
//   W(i,j) -= conj(W(k,i)) W(k,j) / p_k    k < i <= j   (trailing Schur complement)
//   T(i,j) -= T(i,k) W(k,j) / p_k          i < k < j
//   T(k,j)  = W(k,j) / p_k                 j > k         (row k becomes X(k,k) R(k,j))
// with p_k = W(k,k): a rank-1 update of every column right of k.  The two
// index ranges occupy disjoint rows of a column (rows <= k hold T, rows > k
// hold W), and at the end X(i,j) = -T(i,j) / R(j,j), X(j,j) = 1 / R(j,j).
//
// Eight steps go together, so that the chain of barriers is one eighth as
// long: column block K (8 columns, on CTA K mod P of a cluster that keeps
// the packed upper triangle in its shared memory)
//   1. its owner eliminates inside the block: one warp the 8 x 8 diagonal
//      block, then one thread per row the rows above it;
//   2. one thread per remaining column runs the eight pivot rows through the
//      diagonal block (forward substitution), which gives the column's eight
//      factors c_l and its entries of the block's rows;
//   3. with F(l,i) = T(i, k0+l) above the block and conj W(k0+l, i) right of
//      it, every remaining element loses sum_l F(l,i) c_l(j).
// The panel F and the diagonal block travel through global memory (L2): one
// writer and many readers, where pushes through distributed shared memory
// cost 6-8 cycles per 16 bytes and target.  Two cluster barriers per block.
// *status = 1 if a pivot was not finite or, with floor 0, not positive.
//
// Bound by the chain: about 4 us a block.  Measured per solve at orders
// around 120 (12-atom cell, B200): one CTA with the packed triangle, one
// column per step, 281 us; a cluster with one column per step 235 us; this
// kernel 135 us.
//
// Orders beyond a cluster (kGrid, cooperative launch): the same sweep over the
// CTAs of the whole GPU, column block K on CTA K mod P, bounded grid barriers.
// The panel (8 m elements) does not fit beside the columns there: a thread
// takes rows of all the CTA's columns and reads their eight panel elements
// from L2 once.  The 17 pencils of orders 434 to 1,200 of a 480-band solve:
// 26.6 ms (10 us a block: two grid barriers, the owner's elimination, the
// update); with that solve at 561 ms, 577 with cuSOLVER's zpotrf and three ztrsm in
// place of this kernel and three products.
constexpr int kClThreads = 256;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClCols = 4;                        // columns a warp carries at once
constexpr int kFB = 8;                            // columns per block of the metric factor
constexpr double kPivotFloor = 1.0e-14;           // of the unit scaled diagonal

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Barrier of the P CTAs working on one matrix.
__device__ __forceinline__ void group_barrier(int P) {
  if (P == 1) {
    __syncthreads();
  } else {
    cluster_arrive();
    cluster_wait();
  }
}

constexpr unsigned long long kGridWaitNs = 2000000000ull;

__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until `counter` reaches `target`; false when it does not in time or another CTA gave up.
__device__ bool grid_wait(const int* counter, int target, int* err) {
  unsigned long long t0 = 0;
  for (unsigned spin = 0;; ++spin) {
    if (load_acquire(counter) >= target) return true;
    if ((spin & 255u) == 255u) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (t - t0 > kGridWaitNs || *reinterpret_cast<volatile int*>(err) != 0) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
}

// Barrier of a cooperative launch's CTAs; false when it gave up.
__device__ bool grid_barrier(int* counter, int& target, int* err) {
  __shared__ int ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1);
    ok = grid_wait(counter, target, err);
  }
  __syncthreads();
  return ok;
}

// Packed column storage of CTA `rank`: its t-th block (block t P + rank of
// the matrix) starts at this element and keeps 8 columns of 8 (t P + rank + 1) rows.
__host__ __device__ inline size_t factor_base(int t, int P, int rank) {
  return size_t(kFB) * kFB * (size_t(P) * t * (t - 1) / 2 + size_t(t) * (rank + 1));
}

__host__ inline size_t factor_smem(int m, int P, bool grid = false) {
  const int nblk = (m + kFB - 1) / kFB;
  size_t most = 0;
  for (int r = 0; r < P && r < nblk; ++r) most = std::max(most, factor_base((nblk - r + P - 1) / P, P, r));
  const size_t cols = size_t((nblk + P - 1) / P) * kFB;
  return (most + (grid ? 0 : size_t(kFB) * m) + kFB * cols + 3 * kFB * kFB) * sizeof(double2) +
         (2 * size_t(m) + kFB) * sizeof(double);
}

// Global scratch of the factor, in double2: the panel and the diagonal block, by parity of K.
__host__ __device__ inline size_t factor_panel(int m) { return size_t(kFB) * m + 2 * kFB * kFB + kFB; }

// grid_state (kGrid): barrier counter and error flag, zero at launch.
template <bool kGrid>
__global__ void __launch_bounds__(kClThreads) metric_factor_kernel(double2* __restrict__ M, int m, int P,
                                                                   double2* __restrict__ panels,
                                                                   int* __restrict__ status, int* grid_state,
                                                                   double floor) {
  wait_previous();
  const int rank = blockIdx.x;   // the grid is one cluster of P CTAs, or a cooperative launch of P
  const int nblk = (m + kFB - 1) / kFB, nown = nblk > rank ? (nblk - rank + P - 1) / P : 0;
  const int maxown = (nblk + P - 1) / P * kFB;
  extern __shared__ __align__(16) double2 cols[];
  size_t most = 0;
  for (int r = 0; r < P && r < nblk; ++r) {
    const size_t s = factor_base((nblk - r + P - 1) / P, P, r);
    if (s > most) most = s;
  }
  double2* F = cols + most;                                   // [kFB][m]
  double2* sc = F + (kGrid ? 0 : size_t(kFB) * m);            // [kFB][maxown]: c_l of the owned columns
  double2* sW = sc + size_t(kFB) * maxown;                    // [kFB][kFB]: W(k0+l, k0+c) before its scaling
  double2* sC = sW + kFB * kFB;                               // [kFB][kFB]: c(l, c) inside the block
  double2* sD = sC + kFB * kFB;                               // [kFB][kFB]: the block; at the end T inside it
  double* dsc = reinterpret_cast<double*>(sD + kFB * kFB);    // D
  double* ir = dsc + m;                                       // 1 / R(k,k) of the owned columns
  double* sinv = ir + m;                                      // [kFB] 1 / p
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (rank == 0 && tid == 0) *status = 0;   // at least one group barrier lies before another CTA's flag
  for (int j = tid; j < m; j += kClThreads) dsc[j] = 1.0 / sqrt(fmax(M[size_t(j) * m + j].x, DBL_MIN));
  __syncthreads();
  auto column_of = [&](int t, int c) {   // owned column c of block t P + rank
    return cols + factor_base(t, P, rank) + size_t(c) * (size_t(kFB) * (t * P + rank + 1));
  };
  for (int q = warp; q < nown * kFB; q += kClWarps) {
    const int t = q / kFB, c = q - t * kFB, j = (t * P + rank) * kFB + c;
    if (j >= m) continue;
    const double dj = dsc[j];
    double2* col = column_of(t, c);
    for (int i = lane; i <= j; i += 32) {
      double2 v = M[size_t(j) * m + i];
      if (i == j) v.y = 0.0;
      col[i] = cscale(v, dsc[i] * dj);
    }
  }
  __syncthreads();
  int bad = 0, target = 0;
  auto barrier = [&]() {
    if constexpr (kGrid) {
      return grid_barrier(grid_state, target, grid_state + 1);
    } else {
      group_barrier(P);
      return true;
    }
  };
  for (int K = 0; K < nblk; ++K) {
    const int k0 = K * kFB, kb = min(kFB, m - k0), k1 = k0 + kb, owner = K % P;
    double2* panel = panels + (K & 1) * factor_panel(m);
    double2* pdiag = panel + size_t(kFB) * m;   // sW, then T inside the block, then 1 / p
    if (rank == owner) {
      const int t = K / P;
      if (warp == 0) {   // the diagonal block: element (r, c), r <= c, two per lane
        for (int e = lane; e < kFB * kFB; e += 32) {
          const int r = e >> 3, c = e & 7;
          sD[e] = r <= c && c < kb ? column_of(t, c)[k0 + r] : make_double2(0.0, 0.0);
          sW[e] = sC[e] = make_double2(0.0, 0.0);
        }
        __syncwarp();
        for (int l = 0; l < kb; ++l) {
          const double p = sD[l * kFB + l].x;
          const bool dep = !(p > floor);   // also true for NaN
          const double invp = dep ? 0.0 : 1.0 / p;
          double2 out[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int e = lane + 32 * h, r = e >> 3, c = e & 7;
            double2 x = sD[e];
            if (c > l && r <= c && c < kb) {
              const double2 w = sD[l * kFB + c], f = cscale(w, invp);
              if (r == l) {
                x = f;
              } else {
                const double2 a = r < l ? sD[r * kFB + l] : make_double2(sD[l * kFB + r].x, -sD[l * kFB + r].y);
                x = csub(x, cmul(a, f));
              }
            }
            out[h] = x;
          }
          if (lane < kFB && lane > l) {
            sW[l * kFB + lane] = sD[l * kFB + lane];
            sC[l * kFB + lane] = cscale(sD[l * kFB + lane], invp);
          }
          if (lane == 0) {
            if (!isfinite(p) || (dep && floor == 0.0)) bad = 1;
            sinv[l] = invp;
            ir[k0 + l] = p;   // 1 / R(k,k) below
          }
          __syncwarp();
          sD[lane] = out[0];
          sD[lane + 32] = out[1];
          __syncwarp();
        }
        if (lane < kb) {
          const double p = ir[k0 + lane];
          ir[k0 + lane] = !(p > floor) ? 1.0e7 : 1.0 / sqrt(p);
        }
        for (int e = lane; e < kFB * kFB; e += 32) {
          const int r = e >> 3, c = e & 7;
          if (r < c && c < kb) column_of(t, c)[k0 + r] = sD[e];
          if (P > 1) {
            pdiag[e] = sW[e];
            pdiag[kFB * kFB + e] = sD[e];
          }
        }
        if (P > 1 && lane < kb) pdiag[2 * kFB * kFB + lane] = make_double2(sinv[lane], 0.0);
      }
      __syncthreads();
      {
        for (int i = tid; i < k0; i += kClThreads) {   // rows above the block
          double2 tv[kFB];
#pragma unroll
          for (int l = 0; l < kFB; ++l) tv[l] = l < kb ? column_of(t, l)[i] : make_double2(0.0, 0.0);
#pragma unroll
          for (int l = 0; l < kFB; ++l)
#pragma unroll
            for (int c = l + 1; c < kFB; ++c) tv[c] = csub(tv[c], cmul(tv[l], sC[l * kFB + c]));
#pragma unroll
          for (int l = 0; l < kFB; ++l)
            if (l < kb) {
              column_of(t, l)[i] = tv[l];
              if (P > 1) panel[size_t(l) * m + i] = tv[l];
              else F[size_t(l) * m + i] = tv[l];
            }
        }
      }
    }
    if (k1 >= m) break;   // the last block has no columns to its right
    if (!barrier()) {
      if (tid == 0) atomicExch(status, kWaitGaveUp);
      return;
    }
    if (rank != owner) {
      for (int e = tid; e < kFB * kFB; e += kClThreads) {
        sW[e] = __ldcg(pdiag + e);
        sD[e] = __ldcg(pdiag + kFB * kFB + e);
      }
      if (tid < kFB) sinv[tid] = __ldcg(pdiag + 2 * kFB * kFB + tid).x;
      __syncthreads();
    }
    // owned columns right of the block, one thread each (a full block: kb = kFB)
    const int t0 = K + 1 > rank ? (K + 1 - rank + P - 1) / P : 0;   // first owned block right of K
    for (int q = t0 * kFB + tid; q < nown * kFB; q += kClThreads) {
      const int t = q / kFB, c = q - t * kFB, j = (t * P + rank) * kFB + c;
      if (j >= m) continue;
      double2* col = column_of(t, c) + k0;
      double2 y[kFB], f[kFB];
#pragma unroll
      for (int l = 0; l < kFB; ++l) y[l] = col[l];
#pragma unroll
      for (int l = 0; l < kFB; ++l) {
        f[l] = cscale(y[l], sinv[l]);
#pragma unroll
        for (int r = l + 1; r < kFB; ++r) y[r] = csub(y[r], cconjmul(sW[l * kFB + r], f[l]));
      }
#pragma unroll
      for (int l = 0; l < kFB; ++l) {
        sc[size_t(l) * maxown + q] = f[l];
        const double2 w = make_double2(y[l].x, -y[l].y);
        if (P > 1) panel[size_t(l) * m + j] = w;
        else F[size_t(l) * m + j] = w;
        double2 tv = f[l];
#pragma unroll
        for (int r = l + 1; r < kFB; ++r) tv = csub(tv, cmul(sD[l * kFB + r], f[r]));
        col[l] = tv;
      }
    }
    if (!barrier()) {
      if (tid == 0) atomicExch(status, kWaitGaveUp);
      return;
    }
    if constexpr (kGrid) {
      const int last = nown > t0 ? min(m, ((nown - 1) * P + rank + 1) * kFB) : 0;   // rows of the longest column
      for (int i = tid; i < last; i += kClThreads) {
        if (i >= k0 && i < k1) continue;
        double2 f[kFB];
#pragma unroll
        for (int l = 0; l < kFB; ++l) f[l] = __ldcg(panel + size_t(l) * m + i);
        for (int t = t0; t < nown; ++t) {
          const int j0 = (t * P + rank) * kFB;
          double2* col = column_of(t, 0) + i;
          const int stride = kFB * (t * P + rank + 1);
#pragma unroll 4
          for (int c = 0; c < kFB; ++c) {
            if (i <= j0 + c && j0 + c < m) {
              double2 x = col[size_t(c) * stride];
#pragma unroll
              for (int l = 0; l < kFB; ++l) {
                const double2 g = sc[size_t(l) * maxown + t * kFB + c];
                x.x -= f[l].x * g.x - f[l].y * g.y;
                x.y -= f[l].x * g.y + f[l].y * g.x;
              }
              col[size_t(c) * stride] = x;
            }
          }
        }
      }
      __syncthreads();
      continue;
    }
    if (P > 1) {
      for (int e = tid; e < kFB * m; e += kClThreads) {
        const int i = e % m;
        if (i < k0 || i >= k1) F[e] = __ldcg(panel + e);
      }
      __syncthreads();
    }
    for (int q0 = t0 * kFB + warp; q0 < nown * kFB; q0 += kClWarps * kClCols) {
      int jj[kClCols];
      double2* col[kClCols];
      int jmax = -1;
#pragma unroll
      for (int u = 0; u < kClCols; ++u) {
        const int q = q0 + u * kClWarps, t = q / kFB, c = q - t * kFB;
        const int j = (t * P + rank) * kFB + c;
        jj[u] = q < nown * kFB && j < m ? j : -1;
        col[u] = jj[u] >= 0 ? column_of(t, c) : cols;
        jmax = max(jmax, jj[u]);
      }
      for (int i = lane; i <= jmax; i += 32) {
        if (i >= k0 && i < k1) continue;
        double2 f[kFB];
#pragma unroll
        for (int l = 0; l < kFB; ++l) f[l] = F[size_t(l) * m + i];
#pragma unroll
        for (int u = 0; u < kClCols; ++u) {
          if (i <= jj[u]) {
            double2 x = col[u][i];
#pragma unroll
            for (int l = 0; l < kFB; ++l) {
              const double2 c = sc[size_t(l) * maxown + q0 + u * kClWarps];
              x.x -= f[l].x * c.x - f[l].y * c.y;
              x.y -= f[l].x * c.y + f[l].y * c.x;
            }
            col[u][i] = x;
          }
        }
      }
    }
    __syncthreads();
  }
  __syncthreads();
  // U = D X with X(i,j) = -T(i,j) / R(j,j), X(j,j) = 1 / R(j,j); lower triangle zero
  for (int q = warp; q < nown * kFB; q += kClWarps) {
    const int t = q / kFB, c = q - t * kFB, j = (t * P + rank) * kFB + c;
    if (j >= m) continue;
    const double irj = ir[j];
    const double2* col = column_of(t, c);
    for (int i = lane; i < m; i += 32) {
      double2 u = make_double2(0.0, 0.0);
      if (i < j) u = cscale(col[i], -irj * dsc[i]);
      else if (i == j) u = make_double2(irj * dsc[i], 0.0);
      M[size_t(j) * m + i] = u;
    }
  }
  if (bad) atomicExch(status, 1);
}

__host__ __device__ inline size_t hetrd_smem(int n, int p) {
  return (size_t((n + p - 1) / p) * n + 6 * size_t(n)) * sizeof(double2);
}

// Householder reduction of a Hermitian A (n x n, upper triangle read) to the
// real tridiagonal T = Q^H A Q, in the storage convention of LAPACK zhetrd
// with UPLO = 'U' (the published zhetd2 algorithm): for i = n-2 .. 0 the
// reflector H(i) = I - tau_i v v^H with v(i) = 1 and v(0:i-1) left in
// A(0:i-1, i+1) annihilates A(0:i-1, i+1); d = diag(T), e = superdiagonal.
//
// One cluster of CTAs holds the whole (both triangles) matrix in its shared
// memory, column j on CTA j mod P, so a product with A is one local dot
// product per column.  The step is bound by its chain of barriers and
// reductions, so it is arranged around one block and one cluster barrier:
// * the pass over the columns applies the previous step's rank-2 update and
//   forms u = A x with the unnormalised pivot column x, whose norm every warp
//   sums on the way; with v = sc x + kappa e(i), kappa = 1 - sc x(i), the
//   product the method needs is  A v = sc u + kappa A(:, i);
// * each warp pushes its entries of u to every CTA, and forms tau, sc and
//   kappa while the cluster barrier completes;
// * then every CTA pulls column i from its owner and has all it needs:
//   q = x^H u,  y = tau A v,  v^H A v = |sc|^2 q + 2 Re(conj(sc) kappa conj(u(i))) +
//   |kappa|^2 A(i,i),  w = y - (|tau|^2 v^H A v / 2) v  and the next pivot
//   column A(:, i) - v conj(w(i)) - w.
// All CTAs do the same arithmetic in the same order, so their copies agree
// bit for bit.  Measured per solve at orders around 120 (12-atom cell, B200):
// one CTA with the packed triangle 689 us; this kernel with three more block
// barriers per step (norm, v and y^H v) 307 us; as it stands 270 us.
constexpr int kTrdRows = 2;                        // rows of a vector per thread
static_assert(SmallEigen::kOwnMaxOrder <= kTrdRows * kClThreads, "rows of a vector per thread");

__global__ void __launch_bounds__(kClThreads) hetrd_kernel(double2* __restrict__ A, int n, double* __restrict__ dout,
                                                           double* __restrict__ eout, double2* __restrict__ tauout) {
  wait_previous();
  cg::cluster_group cl = cg::this_cluster();
  const int P = int(cl.num_blocks()), rank = int(cl.block_rank());   // P is a power of two
  const int lg = 31 - __clz(P);
  const int nc = (n + P - 1) / P;
  extern __shared__ __align__(16) double2 cols[];   // nc x n: column jl P + rank at cols + jl n
  double2* ubuf = cols + size_t(nc) * n;            // 2 x n: A x, by parity of the step
  double2* xbufs = ubuf + 2 * n;                    // 2 x n: the pivot column
  double2* vbuf = xbufs + 2 * n;                    // n: the previous step's v and w
  double2* wbuf = vbuf + n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int jl = warp; jl * P + rank < n; jl += kClWarps) {
    const int j = jl * P + rank;
    for (int r = lane; r < n; r += 32) {
      double2 a = r <= j ? A[size_t(j) * n + r] : A[size_t(r) * n + j];
      if (r == j) a.y = 0.0;
      if (r > j) a.y = -a.y;
      cols[size_t(jl) * n + r] = a;
    }
  }
  for (int r = tid; r < n; r += kClThreads) vbuf[r] = wbuf[r] = make_double2(0.0, 0.0);
  cl.sync();
  double2 x[kTrdRows];   // the pivot column, rows tid + kClThreads t
  {
    const double2* c = cl.map_shared_rank(cols, (n - 1) & (P - 1)) + size_t((n - 1) >> lg) * n;
#pragma unroll
    for (int t = 0; t < kTrdRows; ++t) {
      const int r = tid + kClThreads * t;
      x[t] = r < n ? c[r] : make_double2(0.0, 0.0);
    }
  }
  int par = 0;
  for (int i0 = n - 2; i0 >= 0; --i0, par ^= 1) {
    const int c = i0 + 1, L = i0 + 1;
    double2* xbuf = xbufs + par * n;
#pragma unroll
    for (int t = 0; t < kTrdRows; ++t) {
      const int r = tid + kClThreads * t;
      if (r < L) xbuf[r] = x[t];
      if (r == c && rank == 0) dout[c] = x[t].x;
    }
    __syncthreads();   // xbuf, vbuf, wbuf
    // columns s < L: the previous rank-2 update, then u(s) = sum_r conj(A(r, s)) x(r)
    double2* u = ubuf + par * n;
    double norm = 0;
    bool first = true;
    int jl0 = warp;
    do {   // at least once: every warp needs the norm
      double2 ws[kClCols], vs[kClCols];
      double acc[2 * kClCols] = {};
      bool on[kClCols];
#pragma unroll
      for (int k = 0; k < kClCols; ++k) {
        const int s = (jl0 + k * kClWarps) * P + rank;
        on[k] = s < L;
        ws[k] = on[k] ? wbuf[s] : make_double2(0.0, 0.0);
        vs[k] = on[k] ? vbuf[s] : make_double2(0.0, 0.0);
      }
      for (int r = lane; r < L; r += 32) {
        const double2 pv = vbuf[r], pw = wbuf[r], xx = xbuf[r];
        if (first && r < i0) norm += xx.x * xx.x + xx.y * xx.y;
#pragma unroll
        for (int k = 0; k < kClCols; ++k) {
          if (on[k]) {
            double2* e = cols + size_t(jl0 + k * kClWarps) * n + r;
            double2 a = *e;
            a.x -= (pv.x * ws[k].x + pv.y * ws[k].y) + (pw.x * vs[k].x + pw.y * vs[k].y);
            a.y -= (pv.y * ws[k].x - pv.x * ws[k].y) + (pw.y * vs[k].x - pw.x * vs[k].y);
            *e = a;
            acc[2 * k] += a.x * xx.x + a.y * xx.y;
            acc[2 * k + 1] += a.x * xx.y - a.y * xx.x;
          }
        }
      }
      first = false;
      const double own = warp_sum8(acc);                                // value lane >> 2
      const double other = __shfl_xor_sync(0xffffffffu, own, 4);
      const bool im = lane & 4;
      const double2 us = make_double2(im ? other : own, im ? own : other);
      const int s = (jl0 + (lane >> 3) * kClWarps) * P + rank;          // eight lanes per column push
      if (s < L) {
        for (int r = lane & 7; r < P; r += 8) cl.map_shared_rank(u, r)[s] = us;
      }
      jl0 += kClWarps * kClCols;
    } while (jl0 * P + rank < L);
    const double2 al = xbuf[i0];
    cluster_arrive();   // this thread is done with v and w in shared memory
    for (int off = 16; off > 0; off >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, off);
    double2 tau = make_double2(0.0, 0.0), sc = make_double2(1.0, 0.0);
    double beta = al.x;
    if (!(norm == 0.0 && al.y == 0.0)) {   // zlarfg on (alpha = x(i0), x(0:i0-1))
      beta = -copysign(sqrt(al.x * al.x + al.y * al.y + norm), al.x);
      const double ib = 1.0 / beta;
      tau = make_double2((beta - al.x) * ib, -al.y * ib);
      const double dr = al.x - beta, di = al.y, iden = 1.0 / (dr * dr + di * di);
      sc = make_double2(dr * iden, -di * iden);   // 1 / (alpha - beta)
    }
    const double2 kap = csub(make_double2(1.0, 0.0), cmul(sc, al));
    const double tau2 = tau.x * tau.x + tau.y * tau.y, sc2 = sc.x * sc.x + sc.y * sc.y;
    const double2 tsc = cmul(tau, sc), tkap = cmul(tau, kap);
    if (rank == 0 && tid == 0) {
      eout[i0] = beta;
      tauout[i0] = tau;
    }
    cluster_wait();
    const double2* next = cl.map_shared_rank(cols, i0 & (P - 1)) + size_t(i0 >> lg) * n;
    double2 ur[kTrdRows], ar[kTrdRows];
#pragma unroll
    for (int t = 0; t < kTrdRows; ++t) {
      const int r = tid + kClThreads * t;
      ar[t] = r <= i0 ? next[r] : make_double2(0.0, 0.0);
      ur[t] = r <= i0 ? u[r] : make_double2(0.0, 0.0);
    }
    const double2 ai = next[i0], ui = u[i0];
    double qs = 0;
    for (int r = lane; r < L; r += 32) {
      const double2 a = xbuf[r], b = u[r];
      qs += a.x * b.x + a.y * b.y;   // Re(conj(x) u)
    }
    for (int off = 16; off > 0; off >>= 1) qs += __shfl_xor_sync(0xffffffffu, qs, off);
    const double2 sk = cconjmul(sc, kap);   // conj(sc) kappa
    const double vav = sc2 * qs + 2.0 * (sk.x * ui.x + sk.y * ui.y) + (kap.x * kap.x + kap.y * kap.y) * ai.x;
    const double a2 = -0.5 * tau2 * vav;
    double2 wi = cadd(cmul(tsc, ui), cmul(tkap, ai));
    wi.x += a2;   // w(i0), v(i0) = 1
#pragma unroll
    for (int t = 0; t < kTrdRows; ++t) {
      const int r = tid + kClThreads * t;
      if (r <= i0) {
        const double2 v = r < i0 ? cmul(x[t], sc) : make_double2(1.0, 0.0);
        if (r < i0 && rank == (c & (P - 1))) A[size_t(c) * n + r] = v;
        double2 w = cadd(cmul(tsc, ur[t]), cmul(tkap, ar[t]));
        w.x += a2 * v.x;
        w.y += a2 * v.y;
        vbuf[r] = v;
        wbuf[r] = w;
        x[t].x = ar[t].x - (v.x * wi.x + v.y * wi.y) - w.x;
        x[t].y = ar[t].y - (v.y * wi.x - v.x * wi.y) - w.y;
      }
    }
  }
  if (rank == 0 && tid == 0) dout[0] = x[0].x;
  cl.sync();   // no CTA leaves while another may still read its columns
}

// The same reduction for orders beyond one cluster: a cooperative launch of
// one CTA per SM, column j on CTA j mod G, u and the pivot column exchanged
// through global memory (L2), one grid barrier per step.  Waits are bounded:
// a barrier that is not reached in two seconds raises *err, and every CTA
// leaves.  Needs ceil(n / G) n elements of shared memory per CTA.
//
// Bound by the chain per step (grid barrier, L2 round trips, reductions) and,
// near the upper end, by the pass over shared memory.  A thread owns rows
// tid + 256 t of all the CTA's columns, so that x, v and w of its rows stay in
// registers and the pass reads and writes each element once and nothing else;
// with a warp per column the three vectors came from shared memory for every
// column (84.5 ms for the 17 pencils of orders 434 to 1,200 of a 480-band
// solve, 63.3 ms like this; cuSOLVER's zhetrd 187 ms for these and the eight
// smaller ones, which take 10.4 ms in the cluster kernel).
constexpr int kGridRows = (SmallEigen::kGridMaxOrder + kClThreads - 1) / kClThreads;
constexpr int kGridCols = 12;   // columns a CTA can own, a multiple of kClCols

inline size_t hetrd_grid_smem(int n, int ctas) {
  return size_t((n + ctas - 1) / ctas) * n * sizeof(double2);
}

// exchange: u and the pivot column, 2 x 2 x n by parity of the step; counter
// zero at launch.
__global__ void __launch_bounds__(kClThreads) hetrd_grid_kernel(double2* __restrict__ A, int n,
                                                                double* __restrict__ dout, double* __restrict__ eout,
                                                                double2* __restrict__ tauout, double2* exchange,
                                                                int* counter, int* err) {
  const int G = gridDim.x, rank = blockIdx.x;
  extern __shared__ __align__(16) double2 cols[];   // ceil(n / G) x n: column jl G + rank at cols + jl n
  __shared__ double red[kClWarps][2 * kGridCols];   // the warps' shares of u
  __shared__ double rnorm[kClWarps], rqs[kClWarps];
  __shared__ double2 vcol[kGridCols], wcol[kGridCols];   // the previous step's v and w at this CTA's columns
  __shared__ double2 s_al;
  __shared__ int s_ok;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int jl = warp; jl * G + rank < n; jl += kClWarps) {
    const int j = jl * G + rank;
    for (int r = lane; r < n; r += 32) {
      double2 a = r <= j ? A[size_t(j) * n + r] : A[size_t(r) * n + j];
      if (r == j) a.y = 0.0;
      if (r > j) a.y = -a.y;
      cols[size_t(jl) * n + r] = a;
    }
  }
  if (tid < kGridCols) vcol[tid] = wcol[tid] = make_double2(0.0, 0.0);
  // rows tid + kClThreads t: the pivot column, the previous step's v and w
  double2 x[kGridRows], v[kGridRows], w[kGridRows];
  int slot[kGridRows];   // row r is this CTA's column slot, or -1
#pragma unroll
  for (int t = 0; t < kGridRows; ++t) {
    const int r = tid + kClThreads * t;
    x[t] = r < n ? A[size_t(n - 1) * n + r] : make_double2(0.0, 0.0);
    if (r == n - 1) x[t].y = 0.0;
    v[t] = w[t] = make_double2(0.0, 0.0);
    slot[t] = r < n && r % G == rank ? r / G : -1;
  }
  // A is overwritten with the reflectors from the first step on: wait until
  // every CTA has read its columns
  int target = G;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    atomicAdd(counter, 1);
    s_ok = grid_wait(counter, target, err);
  }
  __syncthreads();
  if (!s_ok) return;
  int par = 0;
  for (int i0 = n - 2; i0 >= 0; --i0, par ^= 1) {
    const int c = i0 + 1, L = i0 + 1;
    double2* gu = exchange + size_t(2 * par) * n;
    double2* ga = gu + n;
    double norm = 0;
#pragma unroll
    for (int t = 0; t < kGridRows; ++t) {
      const int r = tid + kClThreads * t;
      if (r < i0) norm += x[t].x * x[t].x + x[t].y * x[t].y;
      if (r == i0) s_al = x[t];
      if (r == c && rank == 0) dout[c] = x[t].x;
    }
    __syncthreads();   // vcol, wcol
    // columns s < L: the previous rank-2 update, then u(s) = sum_r conj(A(r, s)) x(r)
    for (int jl0 = 0; jl0 * G + rank < L; jl0 += kClCols) {
      double acc[2 * kClCols] = {};
#pragma unroll
      for (int k = 0; k < kClCols; ++k) {
        const int s = (jl0 + k) * G + rank;
        if (s < L) {
          const double2 ws = wcol[jl0 + k], vs = vcol[jl0 + k];
          double2* col = cols + size_t(jl0 + k) * n;
#pragma unroll
          for (int t = 0; t < kGridRows; ++t) {
            const int r = tid + kClThreads * t;
            if (r < L) {
              double2 a = col[r];
              a.x -= (v[t].x * ws.x + v[t].y * ws.y) + (w[t].x * vs.x + w[t].y * vs.y);
              a.y -= (v[t].y * ws.x - v[t].x * ws.y) + (w[t].y * vs.x - w[t].x * vs.y);
              col[r] = a;
              if (s == i0) ga[r] = a;
              acc[2 * k] += a.x * x[t].x + a.y * x[t].y;
              acc[2 * k + 1] += a.x * x[t].y - a.y * x[t].x;
            }
          }
        }
      }
      const double sum = warp_sum8(acc);   // value lane >> 2
      if ((lane & 3) == 0) red[warp][2 * jl0 + (lane >> 2)] = sum;
    }
    for (int off = 16; off > 0; off >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, off);
    if (lane == 0) rnorm[warp] = norm;
    const double2 own_al = s_al;   // written before the barrier above
    target += G;
    __syncthreads();   // red, rnorm; this CTA's part of the pivot column is written
    if (warp == 0) {
      const int s = (lane >> 1) * G + rank;
      if (s < L) {   // at most 2 kGridCols <= 32 values
        double sum = red[0][lane];
#pragma unroll
        for (int k = 1; k < kClWarps; ++k) sum += red[k][lane];
        reinterpret_cast<double*>(gu + s)[lane & 1] = sum;
      }
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        atomicAdd(counter, 1);
      }
    }
    norm = rnorm[0];
#pragma unroll
    for (int k = 1; k < kClWarps; ++k) norm += rnorm[k];
    const double2 al = own_al;
    double2 tau = make_double2(0.0, 0.0), sc = make_double2(1.0, 0.0);
    double beta = al.x;
    if (!(norm == 0.0 && al.y == 0.0)) {   // zlarfg on (alpha = x(i0), x(0:i0-1))
      beta = -copysign(sqrt(al.x * al.x + al.y * al.y + norm), al.x);
      const double ib = 1.0 / beta;
      tau = make_double2((beta - al.x) * ib, -al.y * ib);
      const double dr = al.x - beta, di = al.y, iden = 1.0 / (dr * dr + di * di);
      sc = make_double2(dr * iden, -di * iden);   // 1 / (alpha - beta)
    }
    const double2 kap = csub(make_double2(1.0, 0.0), cmul(sc, al));
    const double tau2 = tau.x * tau.x + tau.y * tau.y, sc2 = sc.x * sc.x + sc.y * sc.y;
    const double2 tsc = cmul(tau, sc), tkap = cmul(tau, kap);
    if (rank == 0 && tid == 0) {
      eout[i0] = beta;
      tauout[i0] = tau;
    }
    if (tid == 0) s_ok = grid_wait(counter, target, err);
    __syncthreads();
    if (!s_ok) return;
    double2 ur[kGridRows], ar[kGridRows];
    double qs = 0;
#pragma unroll
    for (int t = 0; t < kGridRows; ++t) {
      const int r = tid + kClThreads * t;
      ur[t] = ar[t] = make_double2(0.0, 0.0);
      if (r <= i0) {
        ur[t] = __ldcg(gu + r);
        ar[t] = __ldcg(ga + r);
      }
    }
    const double2 ui = __ldcg(gu + i0), ai = __ldcg(ga + i0);
#pragma unroll
    for (int t = 0; t < kGridRows; ++t) {
      const int r = tid + kClThreads * t;
      if (r <= i0) qs += x[t].x * ur[t].x + x[t].y * ur[t].y;   // Re(conj(x) u)
    }
    for (int off = 16; off > 0; off >>= 1) qs += __shfl_xor_sync(0xffffffffu, qs, off);
    if (lane == 0) rqs[warp] = qs;
    __syncthreads();
    qs = rqs[0];
#pragma unroll
    for (int k = 1; k < kClWarps; ++k) qs += rqs[k];
    const double2 sk = cconjmul(sc, kap);   // conj(sc) kappa
    const double vav = sc2 * qs + 2.0 * (sk.x * ui.x + sk.y * ui.y) + (kap.x * kap.x + kap.y * kap.y) * ai.x;
    const double a2 = -0.5 * tau2 * vav;
    double2 wi = cadd(cmul(tsc, ui), cmul(tkap, ai));
    wi.x += a2;   // w(i0), v(i0) = 1
#pragma unroll
    for (int t = 0; t < kGridRows; ++t) {
      const int r = tid + kClThreads * t;
      if (r <= i0) {
        v[t] = r < i0 ? cmul(x[t], sc) : make_double2(1.0, 0.0);
        if (r < i0 && rank == c % G) A[size_t(c) * n + r] = v[t];
        w[t] = cadd(cmul(tsc, ur[t]), cmul(tkap, ar[t]));
        w[t].x += a2 * v[t].x;
        w[t].y += a2 * v[t].y;
        if (slot[t] >= 0) {
          vcol[slot[t]] = v[t];
          wcol[slot[t]] = w[t];
        }
        x[t].x = ar[t].x - (v[t].x * wi.x + v[t].y * wi.y) - w[t].x;
        x[t].y = ar[t].y - (v[t].y * wi.x - v[t].x * wi.y) - w[t].y;
      }
    }
  }
  if (rank == 0 && tid == 0) dout[0] = x[0].x;
}

// Orders whose congruence and final rotation go through the block kernels
// (blockops.h) instead of ZGEMM with its split-K reductions: two to four
// launches fewer, while one product does not fill the GPU.
constexpr int kSmallProducts = 176;

constexpr size_t kGridSmem = 227 * 1024 - 2560;   // leaves room for the kernel's static shared memory

// CTAs of the cluster for an order-n tridiagonalisation: measured best at 8
// from order 40 to 176 (order 80: 1, 2, 4, 8 and 16 CTAs 283, 218, 192, 183
// and 191 us); beyond, the shared memory of 16.
int hetrd_ctas(int n) { return n <= 40 ? 4 : n <= 176 ? 8 : 16; }

// CTAs for an order-m metric factor: one while its panel update is short.
int factor_ctas(int m) { return m <= 64 ? 1 : m <= 176 ? 8 : 16; }

// And over the whole GPU: one per column block, at most one per SM.
int factor_grid_ctas(const Runtime& rt, int m) { return std::min(rt.sms, ceil_div(m, kFB)); }

// Launch of one cluster of `ctas` CTAs.
struct ClusterLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  template <typename... KArgs>
  ClusterLaunch(void (*kernel)(KArgs...), int ctas, size_t smem, cudaStream_t s) {
    raise_smem_limit(kernel, smem);
    if (ctas > 8) HALF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as launch_chained
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
  }
  ClusterLaunch(const ClusterLaunch&) = delete;
};

template <typename... KArgs, typename... Args>
void launch_cluster(void (*kernel)(KArgs...), int ctas, size_t smem, cudaStream_t s, Args... args) {
  ClusterLaunch l(kernel, ctas, smem, s);
  HALF_CUDA(cudaLaunchKernelEx(&l.cfg, kernel, args...));
}

template <typename... KArgs>
bool cluster_fits(void (*kernel)(KArgs...), int ctas, size_t smem) {
  ClusterLaunch l(kernel, ctas, smem, nullptr);
  l.cfg.numAttrs = 1;   // the cluster's size alone
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &l.cfg) == cudaSuccess) return clusters > 0;
  cudaGetLastError();
  return false;
}

template <typename... KArgs>
bool block_fits(void (*kernel)(KArgs...), size_t smem) {
  raise_smem_limit(kernel, smem);
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, kClThreads, smem) == cudaSuccess) return blocks > 0;
  cudaGetLastError();
  return false;
}

std::atomic<int> g_cluster_limit{16};
std::atomic<bool> g_grid_limit{true};

// Asks the device, once per runtime, what the pencil kernels can be launched with.
void ask_pencil_limits(Runtime& rt) {
  if (rt.cluster_ctas >= 0) return;
  rt.cluster_ctas = 0;
  for (const auto [ctas, order] : {std::pair(16, SmallEigen::kOwnMaxOrder), std::pair(8, 176), std::pair(4, 40)}) {
    if (ctas > g_cluster_limit.load()) continue;
    if (cluster_fits(hetrd_kernel, ctas, hetrd_smem(order, ctas)) &&
        cluster_fits(metric_factor_kernel<false>, factor_ctas(order), factor_smem(order, factor_ctas(order)))) {
      rt.cluster_ctas = ctas;
      break;
    }
  }
  rt.grid_pencils = g_grid_limit.load() && block_fits(hetrd_grid_kernel, kGridSmem) &&
                    block_fits(metric_factor_kernel<true>, kSmemMax);
}

// A cooperative launch; false (nothing launched, and not tried again on this
// runtime) where the process may not use as many SMs at once.
bool launch_grid(Runtime& rt, const void* kernel, int ctas, void** args, size_t smem) {
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(kClThreads), args, smem, rt.stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    rt.grid_pencils = false;
    return false;
  }
  HALF_CUDA(e);
  rt.prof.launches += 1;
  return true;
}

constexpr int kUnpolishedOrder = 164;

// g = 3/2 - g / 2
__global__ void polish_matrix_kernel(double* __restrict__ g, int n) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < (long long)n * n) g[t] = (t % (n + 1) == 0 ? 1.5 : 0.0) - 0.5 * g[t];
}

__global__ void real_to_complex_block_kernel(const double* __restrict__ z, long long count, double2* __restrict__ out) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < count) out[t] = make_double2(z[t], 0.0);
}

// Large orders (the dense solves): the scaled T stays in global memory, read
// through L1 with all lanes of a warp at the same index.  This kernel scales
// d in place, squares e into e2 and leaves the scaled Gershgorin bounds
// (lo, hi, norm) and the scale in bounds.
__global__ void tridiag_bounds_kernel(double* __restrict__ d, const double* __restrict__ e, int n,
                                      double* __restrict__ e2, double* __restrict__ bounds) {
  __shared__ double s_norm;
  if (threadIdx.x < 32) {
    double gl, gu, nrm;
    gershgorin(d, e, n, gl, gu, nrm);
    if (threadIdx.x == 0) {
      const double sc = norm_scale(nrm);
      s_norm = nrm;
      bounds[0] = gl * sc;
      bounds[1] = gu * sc;
      bounds[2] = nrm * sc;
      bounds[3] = sc;
    }
  }
  __syncthreads();
  const double sc = norm_scale(s_norm);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] *= sc;
    e2[i] = scaled_e2(i < n - 1 ? e[i] : 0.0, sc);
  }
}

// Eigenvalues k0 .. k0 + ne - 1 of T (ascending), one warp each, by the same
// multisection as tridiag_values_kernel.
__global__ void __launch_bounds__(32 * kValueWarps) tridiag_values_global_kernel(const double* __restrict__ d,
                                                                                 const double* __restrict__ e2, int n,
                                                                                 int k0, int ne,
                                                                                 const double* __restrict__ bounds,
                                                                                 double* __restrict__ lam) {
  const int j = blockIdx.x * kValueWarps + (threadIdx.x >> 5);
  if (j >= ne) return;
  const double v = multisect(d, e2, n, k0 + j, bounds[0], bounds[1], bounds[2]);
  if ((threadIdx.x & 31) == 0) lam[j] = v / bounds[3];
}

}  // namespace

std::string pencil_failure(const int* infos) {
  if (infos[1] == kWaitGaveUp || infos[2] == kWaitGaveUp)
    return "ACC small generalized eigensolve: a grid-wide kernel gave up waiting for its other thread blocks";
  if (infos[0] != 0) return "ACC correction metric eigensolve failed (info " + std::to_string(infos[0]) + ")";
  if (infos[2] != 0)
    return "ACC Rayleigh-Ritz overlap is not positive definite (Cholesky info " + std::to_string(infos[2]) + ")";
  if (infos[1] != 0) return "ACC small generalized eigensolve failed (info " + std::to_string(infos[1]) + ")";
  return "";
}

void SmallEigen::reserve(Runtime& rt, int nmax) {
  if (nmax <= cap) return;
  cap = nmax;
  d.resize(nmax);
  e.resize(nmax);
  tau.resize(nmax);
  V.resize(size_t(nmax) * nmax);
  Z.resize(size_t(nmax) * nmax);
  // global inverse-iteration scratch: one slot per thread of the vector kernel's grid
  const size_t slots = size_t(ceil_div(nmax, kVectorThreads)) * kVectorThreads;
  scratch.resize(5 * size_t(nmax) * slots + (size_t(nmax) * slots + 7) / 8 + 16);
  lam.resize(nmax);
  info.resize(1);
  info.zero(rt.stream);
  int l1 = 0, l2 = 0;
  cusolver_check(cusolverDnZhetrd_bufferSize(rt.solver, CUBLAS_FILL_MODE_UPPER, nmax,
                                             reinterpret_cast<cuDoubleComplex*>(V.get()), nmax, d.get(), e.get(),
                                             reinterpret_cast<cuDoubleComplex*>(tau.get()), &l1),
                 "zhetrd buffer");
  cusolver_check(cusolverDnZpotrf_bufferSize(rt.solver, CUBLAS_FILL_MODE_UPPER, nmax,
                                             reinterpret_cast<cuDoubleComplex*>(V.get()), nmax, &l2),
                 "zpotrf buffer");
  int l3 = 0;
  cusolver_check(cusolverDnZunmtr_bufferSize(rt.solver, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, nmax,
                                             nmax, reinterpret_cast<cuDoubleComplex*>(V.get()), nmax,
                                             reinterpret_cast<cuDoubleComplex*>(tau.get()),
                                             reinterpret_cast<cuDoubleComplex*>(V.get()), nmax, &l3),
                 "zunmtr buffer");
  work.resize(size_t(std::max({l1, l2, l3, 1})));
}

void limit_pencil_launches(int cluster_ctas, bool grid) {
  g_cluster_limit.store(cluster_ctas);
  g_grid_limit.store(grid);
}

bool SmallEigen::cluster_order(Runtime& rt, int n) {
  ask_pencil_limits(rt);
  return n <= kOwnMaxOrder && std::max(hetrd_ctas(n), factor_ctas(n)) <= rt.cluster_ctas;
}

bool SmallEigen::grid_order(Runtime& rt, int n) {
  ask_pencil_limits(rt);
  return rt.grid_pencils && n > kOwnMaxOrder && n <= kGridMaxOrder && n <= kGridCols * rt.sms && hetrd_grid_smem(n, rt.sms) <= kGridSmem &&
         factor_smem(n, factor_grid_ctas(rt, n), true) <= kSmemMax;
}

void SmallEigen::clear_grid_state(cudaStream_t s) {
  if (grid_state.size() == 0) grid_state.resize(2);   // barrier counter, error flag
  grid_state.zero(s);
}

// Hermitian eigenproblem of A (n x n, upper triangle used, destroyed); the nev
// lowest eigenvectors go to V[:, :nev] (leading dimension n), eigenvalues to w.
void SmallEigen::heev(Runtime& rt, double2* A, int n, int nev, double* w, int* status, const int* failed) {
  reserve(rt, n);
  cudaStream_t s = rt.stream;
  const int* gave_up = nullptr;
  bool reduced = false;
  if (cluster_order(rt, n)) {   // whole reduction in one cluster
    const int p = hetrd_ctas(n);
    launch_cluster(hetrd_kernel, p, hetrd_smem(n, p), s, A, n, d.get(), e.get(), tau.get());
    rt.prof.launches += 1;
    reduced = true;
  } else if (grid_order(rt, n)) {
    const size_t gsm = hetrd_grid_smem(n, rt.sms);
    if (exchange.size() < 4 * size_t(n)) exchange.resize(4 * size_t(kGridMaxOrder));
    clear_grid_state(s);
    gave_up = grid_state.get() + 1;
    raise_smem_limit(hetrd_grid_kernel, kGridSmem);   // static and dynamic together may pass 48 KB before gsm does
    double *dp = d.get(), *ep = e.get();
    double2 *tp = tau.get(), *xp = exchange.get();
    int *cp = grid_state.get(), *gp = cp + 1;
    void* args[] = {&A, &n, &dp, &ep, &tp, &xp, &cp, &gp};
    reduced = launch_grid(rt, reinterpret_cast<const void*>(hetrd_grid_kernel), rt.sms, args, gsm);
  }
  if (!reduced) {
    gave_up = nullptr;
    cusolver_check(cusolverDnZhetrd(rt.solver, CUBLAS_FILL_MODE_UPPER, n, reinterpret_cast<cuDoubleComplex*>(A), n,
                                    d.get(), e.get(), reinterpret_cast<cuDoubleComplex*>(tau.get()),
                                    reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()), info.get()),
                   "zhetrd");
  }
  // Eigenvalues up to ne = nev + kExtraEig are located so that a cluster
  // straddling the last wanted index is computed (and orthogonalised) whole;
  // only the first nev pairs are returned.
  const int ne = std::min(n, nev + kExtraEig);
  const size_t vsm = 3 * size_t(n) * sizeof(double);
  raise_smem_limit(tridiag_values_kernel, vsm);
  launch_chained(ceil_div(ne, kValueWarps), 32 * kValueWarps, vsm, s, tridiag_values_kernel,
      d.get(), e.get(), n, ne, lam.get(), gave_up, status);
  HALF_LAUNCH("tridiagonal eigenvalues");
  size_t tsm = (2 * size_t(n) + ne) * sizeof(double) + size_t(ne) * sizeof(int);
  if (tsm > kSmemMax) fail(kCapacity, "subspace eigenproblem too large for the tridiagonal solver: n=" + std::to_string(n));
  tsm = (tsm + 15) & ~size_t(15);
  const size_t slot = 5 * size_t(n) * sizeof(double) + size_t(n);
  int per = kVectorThreads;
  while (per > 4 && tsm + per * slot > kSmemMax) per /= 2;
  double* gs = nullptr;
  if (tsm + per * slot <= kSmemMax) {
    tsm += per * slot;
  } else {
    gs = scratch.get();
    per = kVectorThreads;
  }
  raise_smem_limit(tridiag_vectors_kernel, tsm);
  launch_chained(ceil_div(nev, per), kVectorThreads, tsm, s, tridiag_vectors_kernel,
      d.get(), e.get(), n, nev, ne, per, lam.get(), w, Z.get(), gs, status, failed);
  HALF_LAUNCH("tridiagonal eigenvectors");
  // Inverse iteration leaves |<z_i, z_j>| <= eps ||T|| / gap between clusters:
  // 1e-13 in the 12-atom cell's wide blocks, 1e-9 at worst.  One step of
  // Z <- Z (3/2 - Z^T Z / 2) brings that to rounding, which is what cuSOLVER
  // gave the orders above 164 (25 us of a pencil's 1.5 ms and more).
  const double* z = Z.get();
  if (n > kUnpolishedOrder) {
    double* const g = scratch.get();
    double* const z2 = g + size_t(nev) * nev;
    const double one = 1.0, zero = 0.0;
    cublas_check(cublasDgemm(rt.blas, CUBLAS_OP_T, CUBLAS_OP_N, nev, nev, n, &one, z, n, z, n, &zero, g, nev), "dgemm");
    polish_matrix_kernel<<<ceil_div((long long)nev * nev, 256), 256, 0, s>>>(g, nev);
    HALF_LAUNCH("tridiagonal eigenvector overlaps");
    cublas_check(cublasDgemm(rt.blas, CUBLAS_OP_N, CUBLAS_OP_N, n, nev, nev, &one, z, n, g, nev, &zero, z2, n), "dgemm");
    rt.prof.launches += 1;
    z = z2;
  }
  if (n > kOwnMaxOrder) {
    // large orders: cuSOLVER's blocked back-transformation (zunmtr, Q Z with
    // zhetrd's reflectors) on the complex copy of Z
    real_to_complex_block_kernel<<<ceil_div((long long)n * nev, 256), 256, 0, s>>>(z, (long long)n * nev, V.get());
    HALF_LAUNCH("tridiagonal eigenvectors to complex");
    cusolver_check(cusolverDnZunmtr(rt.solver, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, n, nev,
                                    reinterpret_cast<cuDoubleComplex*>(A), n,
                                    reinterpret_cast<cuDoubleComplex*>(tau.get()),
                                    reinterpret_cast<cuDoubleComplex*>(V.get()), n,
                                    reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()), info.get()),
                   "zunmtr");
    rt.prof.launches += 3;
    return;
  }
  // back-transformation: as many reflectors at a time as fit, in blocks of four
  const size_t per_block = kBackBlock * (size_t(n) + 1) * sizeof(double2) + 8 * sizeof(double2);
  const int blocks = int(std::min<size_t>(ceil_div(std::max(n - 1, 1), kBackBlock), kSmemMax / per_block));
  const size_t bsm = size_t(blocks) * per_block;
  auto back = [&](auto kernel) {
    raise_smem_limit(kernel, bsm);
    launch_chained(ceil_div(nev, kBackWarps), 32 * kBackWarps, bsm, s, kernel, A, tau.get(), z, n, nev,
                   blocks * kBackBlock, V.get());
  };
  if (n <= 64) back(back_transform_kernel<2>);
  else if (n <= 160) back(back_transform_kernel<5>);
  else if (n <= 288) back(back_transform_kernel<9>);
  else back(back_transform_kernel<14>);
  HALF_LAUNCH("back transformation");
  rt.prof.launches += 3;
}

// Generalized problem A y = lambda B y (itype 1, upper triangles used), B HPD.
// The nev lowest eigenvectors (Y^H B Y = I) overwrite A[:, :nev].
void SmallEigen::hegv(Runtime& rt, double2* A, double2* B, int n, int nev, double* w, int* status, int* chol_status,
                      bool strict) {
  reserve(rt, n);
  cudaStream_t s = rt.stream;
  bool factored = false;
  if (cluster_order(rt, n)) {
    factored = metric_normalize(rt, B, n, chol_status, strict);
  } else if (grid_order(rt, n)) {
    int p = factor_grid_ctas(rt, n);
    const size_t fsm = factor_smem(n, p, true);
    if (panels.size() < 2 * factor_panel(n)) panels.resize(2 * factor_panel(kGridMaxOrder));
    clear_grid_state(s);
    raise_smem_limit(metric_factor_kernel<true>, kSmemMax);
    double2* pp = panels.get();
    int* gp = grid_state.get();
    double floor = strict ? 0.0 : kPivotFloor;
    void* args[] = {&B, &n, &p, &pp, &chol_status, &gp, &floor};
    factored = launch_grid(rt, reinterpret_cast<const void*>(metric_factor_kernel<true>), p, args, fsm);
  }
  if (factored) {
    // B -> X = D R^-1 with X^H B X = I (metric_factor_kernel), C = X^H A X,
    // C V = V Lambda, Y = X V: the same pencil reduction as zhegvd's
    // Cholesky / two triangular solves, with the factor inverted in shared
    // memory and the products done by three GEMMs.  They need products that
    // are accurate element by element: without a metric step a row of A holds
    // tens of eV beside X-P entries as small as the residuals, and X's P
    // columns are as large as those are small.  (Products that hold a row in
    // fixed point relative to its norm, as zcrt.cu does, stop the residuals of
    // 480 to 512 bands of the 12-atom cell at 5e-6 to 4e-5 eV whatever the
    // tolerance; these reach 1e-7 in 9 iterations.)
    launch_chained(ceil_div((long long)n * n, 256), 256, 0, s, hermitian_fill_kernel,
        A, n);
    rt.prof.launches += 1;
    const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
    if (n <= kSmallProducts) {
      double2* const v = V.get();
      const ZBlock ba = {A, n}, bb = {B, n}, bv = {v, n};
      zupdate(rt, n, &ba, B, n, &v, n, 1, 1.0, 0.0, ZRoute::kBlock);
      zgram(rt, n, bb, &bv, &A, 1, n, true, ZRoute::kBlock);
      heev(rt, A, n, nev, w, status, chol_status);
      zupdate(rt, n, &bb, v, n, &A, nev, 1, 1.0, 0.0, ZRoute::kBlock);
      return;
    }
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, n, n, one, A, n, B, n, zero, V.get(), n);
    gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, n, n, n, one, B, n, V.get(), n, zero, A, n);
    heev(rt, A, n, nev, w, status, chol_status);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, nev, n, one, B, n, V.get(), n, zero, A, n);
    return;
  }
  auto* Bc = reinterpret_cast<cuDoubleComplex*>(B);
  auto* Ac = reinterpret_cast<cuDoubleComplex*>(A);
  cusolver_check(cusolverDnZpotrf(rt.solver, CUBLAS_FILL_MODE_UPPER, n, Bc, n,
                                  reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()), chol_status),
                 "zpotrf");
  launch_chained(ceil_div((long long)n * n, 256), 256, 0, s, hermitian_fill_kernel,
      A, n);
  rt.prof.launches += 1;
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0);
  cublas_check(cublasZtrsm(rt.blas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_C, CUBLAS_DIAG_NON_UNIT, n, n,
                           &one, Bc, n, Ac, n),
               "ztrsm");
  cublas_check(cublasZtrsm(rt.blas, CUBLAS_SIDE_RIGHT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT, n, n,
                           &one, Bc, n, Ac, n),
               "ztrsm");
  heev(rt, A, n, nev, w, status, chol_status);
  HALF_CUDA(cudaMemcpyAsync(A, V.get(), size_t(n) * nev * sizeof(double2), cudaMemcpyDeviceToDevice, s));
  cublas_check(cublasZtrsm(rt.blas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT, n, nev,
                           &one, Bc, n, Ac, n),
               "ztrsm");
}

// U with (P U)^H S (P U) = I from M = P^H S P, overwriting M (see
// metric_factor_kernel); false when m is beyond the cluster's shared memory.
bool SmallEigen::metric_normalize(Runtime& rt, double2* M, int m, int* status, bool strict) {
  if (!cluster_order(rt, m)) return false;
  const int p = factor_ctas(m);
  if (panels.size() < 2 * factor_panel(m)) panels.resize(2 * factor_panel(kOwnMaxOrder));
  launch_cluster(metric_factor_kernel<false>, p, factor_smem(m, p), rt.stream, M, m, p, panels.get(), status,
                 static_cast<int*>(nullptr), strict ? 0.0 : kPivotFloor);
  rt.prof.launches += 1;
  return true;
}

void hermitian_eigenvalues_large(Runtime& rt, double2* A, long long n, const std::vector<int>& k0s,
                                 const std::vector<int>& counts, double* lam) {
  if (n > INT32_MAX / 2) fail(kUnavailable, "dense order beyond the tridiagonalisation's range");
  cudaStream_t s = rt.stream;
  const int ni = int(n);
  DeviceBuffer<double> d(ni), e(ni), e2(ni), bounds(4);
  DeviceBuffer<double2> tau(ni);
  DeviceBuffer<int> info(1);
  int lwork = 0;
  cusolver_check(cusolverDnZhetrd_bufferSize(rt.solver, CUBLAS_FILL_MODE_UPPER, ni,
                                             reinterpret_cast<cuDoubleComplex*>(A), ni, d.get(), e.get(),
                                             reinterpret_cast<cuDoubleComplex*>(tau.get()), &lwork),
                 "zhetrd buffer (large)");
  DeviceBuffer<double2> work(size_t(std::max(lwork, 1)));
  cusolver_check(cusolverDnZhetrd(rt.solver, CUBLAS_FILL_MODE_UPPER, ni, reinterpret_cast<cuDoubleComplex*>(A), ni,
                                  d.get(), e.get(), reinterpret_cast<cuDoubleComplex*>(tau.get()),
                                  reinterpret_cast<cuDoubleComplex*>(work.get()), lwork, info.get()),
                 "zhetrd (large)");
  int hinfo = 0;
  HALF_CUDA(cudaMemcpyAsync(&hinfo, info.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  HALF_CUDA(cudaStreamSynchronize(s));
  if (hinfo != 0) fail(kInternal, "Householder tridiagonalisation failed");
  tridiag_bounds_kernel<<<1, 1024, 0, s>>>(d.get(), e.get(), ni, e2.get(), bounds.get());
  HALF_LAUNCH("tridiagonal bounds");
  int off = 0;
  for (size_t r = 0; r < k0s.size(); ++r) {
    const int k0 = k0s[r], ne = counts[r];
    if (k0 < 0 || ne < 0 || k0 + ne > ni) fail(kInvalidArgument, "eigenvalue index range outside the matrix");
    if (ne == 0) continue;
    tridiag_values_global_kernel<<<ceil_div(ne, kValueWarps), 32 * kValueWarps, 0, s>>>(d.get(), e2.get(), ni, k0, ne,
                                                                                       bounds.get(), lam + off);
    HALF_LAUNCH("tridiagonal eigenvalues (large)");
    off += ne;
  }
  HALF_CUDA(cudaStreamSynchronize(s));
}

}  // namespace hb
