// The all-band `acc` block eigensolver.
//
// Algorithm: src/half_cuda_iterative_solver.cuf:79-310, step for step:
// unit-vector start at the m lowest-kinetic plane waves in the reference's
// heap order, Rayleigh-Ritz, then per iteration residual norms (the diagonal
// of R^H R), unit seeds for converged bands at plane wave (m+j) mod n,
// preconditioner -R/(|T-eps|+1 eV), H/S application, S-orthogonalisation
// against X, S-metric normalisation through eigh(P^H S P) with the 1e-14
// floor, and a generalized Rayleigh-Ritz on [X P].
//
// B200 differences (same mathematics):
// * the residual is never stored: one warp-reduced kernel produces the column
//   norms, a second builds the preconditioned direction (and the seeds) from
//   H X, S X on the fly; the reference's full m x m Gram GEMM is not formed;
// * Rayleigh-Ritz projects only the blocks zhegvd reads (upper triangle), and
//   the rotations write into ping-pong buffers instead of copy-backs;
// * all workspaces and solver buffers are allocated once per solve, one
//   cuBLAS/cuSOLVER handle lives on the context stream, and the only
//   host<->device traffic per iteration is the m residual norms plus the
//   solver status words (one synchronisation, as in the reference);
// * with the library's own small solvers (eig.cu, the default) the
//   correction directions are S-normalised by a Jacobi-scaled Cholesky
//   factor (pivots floored at 1e-14; orders to 164) instead of the
//   eigenvectors of the metric; both bases span the same space, so the Rayleigh-Ritz step and
//   the Ritz values are those of the reference up to rounding;
// * precision MIXED runs the iterations on FP32 blocks (FP32 operator,
//   split-bf16 tcgen05 GEMMs from tc_gemm.cu whose projected matrices land
//   directly in FP64, FP64 small eigensolves) until the residual reaches the
//   FP32 regime, then promotes X
//   and finishes with FP64 iterations (one FP64 operator sweep re-creates
//   H X and S X exactly before the first FP64 Rayleigh-Ritz); it carries
//   m/4 (at least 4) guard bands and tests convergence on the requested m.
#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <string>

#include "blas.h"
#include "blockops.h"
#include "context.h"
#include "eig.h"

namespace hb {

namespace {

// Heap order of src/half_cuda_iterative_solver.cuf:277-310 (0-based output).
std::vector<int> kinetic_order(const std::vector<double>& kin) {
  int n = int(kin.size());
  std::vector<int> ind(n + 1);
  for (int i = 1; i <= n; ++i) ind[i] = i;
  auto K = [&](int i) { return kin[ind[i] - 1]; };
  for (int i = 2; i <= n; ++i) {
    int child = i;
    while (child > 1) {
      int parent = child / 2;
      if (K(parent) >= K(child)) break;
      std::swap(ind[parent], ind[child]);
      child = parent;
    }
  }
  for (int last = n; last >= 2; --last) {
    std::swap(ind[1], ind[last]);
    int parent = 1;
    while (true) {
      int child = 2 * parent;
      if (child > last - 1) break;
      if (child + 1 <= last - 1 && K(child + 1) > K(child)) ++child;
      if (K(parent) >= K(child)) break;
      std::swap(ind[parent], ind[child]);
      parent = child;
    }
  }
  std::vector<int> out(n);
  for (int i = 0; i < n; ++i) out[i] = ind[i + 1] - 1;
  return out;
}

template <typename C>
__global__ void init_states_kernel(C* x, long long ld, int n, int m, const int* idx) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)n * m) return;
  int j = int(t / n), i = int(t - (long long)j * n);
  C v;
  v.x = (i == idx[j]) ? 1 : 0;
  v.y = 0;
  x[(long long)j * ld + i] = v;
}

// norms[j] = || H x_j - eps_j S x_j ||  (one block per band, FP64 accumulation).
// report: what the host reads once per iteration, in one copy: the norms, the
// Ritz values, the three solver status words and the tensor-core error flag.
template <typename C>
__global__ void residual_norm_kernel(const C* __restrict__ hx, const C* __restrict__ sx, long long ld, int n,
                                     const double* __restrict__ eps, const int* __restrict__ info,
                                     const int* __restrict__ tc_err, double* __restrict__ norms,
                                     double* __restrict__ report) {
  after_previous();
  if (blockIdx.x == 0 && threadIdx.x < 4)
    report[2 * gridDim.x + threadIdx.x] =
        threadIdx.x < 3 ? double(info[threadIdx.x]) : tc_err ? double(*tc_err) : 0.0;
  const int j = blockIdx.x;
  const double e = eps[j];
  const C* h = hx + (long long)j * ld;
  const C* s = sx + (long long)j * ld;
  double acc = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double rx = double(h[i].x) - e * double(s[i].x), ry = double(h[i].y) - e * double(s[i].y);
    acc += rx * rx + ry * ry;
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    int nw = blockDim.x >> 5;
    acc = threadIdx.x < nw ? red[threadIdx.x] : 0.0;
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if (threadIdx.x == 0) {
      const double v = sqrt(fmax(0.0, acc));
      norms[j] = v;
      report[j] = v;
      report[gridDim.x + j] = e;
    }
  }
}

// P = -R / (|T - eps| + 1), or the unit seed (m + j) mod n for bands whose
// residual norm is below the seed threshold (src/half_cuda_iterative_solver.cuf:42-64, 150-155)
// Output column a takes band cols[a] (cols null: band a), a < np.
template <typename C, typename CO = C>
__global__ void precondition_kernel(const C* __restrict__ hx, const C* __restrict__ sx, long long ld, int n, int m,
                                    int np, const int* __restrict__ cols, const double* __restrict__ eps,
                                    const double* __restrict__ norms, double seed_threshold,
                                    const double* __restrict__ kinetic, CO* __restrict__ p) {
  after_previous();
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)n * np) return;
  const int a = int(t / n), i = int(t - (long long)a * n);
  const int j = cols ? cols[a] : a;
  long long o = (long long)j * ld + i;
  const long long oa = (long long)a * ld + i;
  CO out;
  if (norms[j] < seed_threshold) {
    int seed = (m + j) % n;
    out.x = (i == seed) ? 1 : 0;
    out.y = 0;
  } else {
    double e = eps[j];
    double den = fabs(kinetic[i] - e) + 1.0;
    out.x = -(double(hx[o].x) - e * double(sx[o].x)) / den;
    out.y = -(double(hx[o].y) - e * double(sx[o].y)) / den;
  }
  p[oa] = out;
}

// U[:, j] /= sqrt(max(mu_j, floor))  (src/half_cuda_iterative_solver.cuf:66-77)
__global__ void scale_columns_kernel(double2* u, int m, const double* mu, double floor_value) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * m) return;
  int j = t / m;
  u[t] = cscale(u[t], 1.0 / sqrt(fmax(mu[j], floor_value)));
}

// Jacobi scaling of an order-n pencil (H, S): d[i] = 1 / sqrt(Re S(i,i))
// (1 where that is not positive) by the first kernel, then H(i,j) and S(i,j)
// times d[i] d[j] by the second.
__global__ void jacobi_diag_kernel(const double2* __restrict__ s, int n, double* __restrict__ d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double si = s[(long long)i * n + i].x;
  d[i] = si > 0.0 ? 1.0 / sqrt(si) : 1.0;
}

__global__ void jacobi_scale_kernel(double2* __restrict__ h, double2* __restrict__ s, int n,
                                    const double* __restrict__ d) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)n * n) return;
  const int i = int(t % n), j = int(t / n);
  const double f = d[i] * d[j];
  h[t] = cscale(h[t], f);
  s[t] = cscale(s[t], f);
}

// Y(i, j) *= d[i] for the first `cols` columns (eigenvectors of the scaled
// pencil back to the unscaled one).
__global__ void scale_rows_kernel(double2* __restrict__ y, int ld, int rows, int cols, const double* __restrict__ d) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)rows * cols) return;
  const int i = int(t % rows), j = int(t / rows);
  y[(long long)j * ld + i] = cscale(y[(long long)j * ld + i], d[i]);
}

// out[:, j] = in[:, perm[j]] for the m columns of an n-row block (ld n).
template <typename C>
__global__ void gather_columns_kernel(const C* __restrict__ in, C* __restrict__ out, int n, int m,
                                      const int* __restrict__ perm) {
  after_previous();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)n * m) return;
  const int j = int(t / n), i = int(t - (long long)j * n);
  out[t] = in[(long long)perm[j] * n + i];
}

__global__ void gather_values_kernel(const double* __restrict__ in, double* __restrict__ out, int m,
                                     const int* __restrict__ perm) {
  after_previous();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) out[j] = in[perm[j]];
}

template <typename A, typename B>
__global__ void convert_kernel(const A* __restrict__ in, B* __restrict__ out, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) {
    B v;
    v.x = in[i].x;
    v.y = in[i].y;
    out[i] = v;
  }
}

// column-major block copy with leading dimensions
template <typename A, typename B>
__global__ void convert_block_kernel(const A* __restrict__ in, long long ldi, B* __restrict__ out, long long ldo,
                                     int rows, int cols) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)rows * cols) return;
  int j = int(t / rows), i = int(t - (long long)j * rows);
  B v;
  v.x = in[j * ldi + i].x;
  v.y = in[j * ldi + i].y;
  out[j * ldo + i] = v;
}

double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// Phase tracer (environment HALF_TRACE=1): synchronises the stream at each
// mark and attributes the elapsed host time to the named phase; the totals go
// to stderr at the end of the solve.  Off by default (no synchronisation).
struct Tracer {
  bool on = std::getenv("HALF_TRACE") != nullptr;
  bool history = on && std::string(std::getenv("HALF_TRACE")) == "2";   // per-iteration residuals
  // res: max residual over the requested bands; also the worst requested band
  // and how many requested bands are at or below lock_tol (soft-locked)
  void step(const char* phase, int it, double res, const std::vector<double>& norms, int mreq, double lock_tol) {
    if (!history) return;
    const int nr = std::min<int>(mreq, int(norms.size()));
    int worst = int(std::max_element(norms.begin(), norms.begin() + nr) - norms.begin());
    int locked = 0;
    for (int j = 0; j < nr; ++j) locked += norms[j] <= lock_tol;
    std::fprintf(stderr, "HALF iter %s %d %.6e band %d locked %d\n", phase, it, res, worst, locked);
  }
  cudaStream_t s = nullptr;
  std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
  std::vector<std::pair<const char*, double>> acc;
  void mark(const char* name) {
    if (!on) return;
    cudaStreamSynchronize(s);
    double d = ms_since(t);
    t = std::chrono::steady_clock::now();
    for (auto& p : acc)
      if (p.first == name) { p.second += d; return; }
    acc.push_back({name, d});
  }
  void report(int iters) {
    if (!on) return;
    std::fprintf(stderr, "HALF trace (%d iterations):", iters);
    for (auto& p : acc) std::fprintf(stderr, " %s=%.2fms", p.first, p.second);
    std::fprintf(stderr, "\n");
  }
};

// FP64 small dense solves on the context's cuSOLVER handle; the status words
// stay on the device and are read with the next residual norms.
// By default the library's own device-resident solvers (eig.cu); environment
// HALF_SMALL_EIG=cusolver selects cuSOLVER zheevd/zhegvd as the reference does.
struct SmallSolver {
  Runtime& rt;
  int m;
  DeviceBuffer<double2> work;
  DeviceBuffer<int> info;   // [0] metric heevd, [1] RR hegvd, [2] RR Cholesky (own solver)
  int lw_ev = 0, lw_gv = 0;
  bool own = true;
  // cuSOLVER pencils: only the nev lowest pairs (zhegvdx, index range; the
  // guard-band modes' default) or all of them (zhegvd: the FP64 mode, or
  // HALF_PENCIL_RANGE=0)
  bool range = true;
  // HALF_PENCIL_OWN=1: pencils above the own solver's order go through
  // SmallEigen::hegv too (cuSOLVER zpotrf / zhetrd / zunmtr around the
  // library's multisection and inverse-iteration kernels)
  bool own_large = false;
  // Above this order the own solver reports an overlap that is not positive
  // definite, as the cuSOLVER calls do that served those orders: the FP64 mode
  // ends with that error, the guard-band modes redo the step with the metric
  // normalisation.  Up to it, it floors the dependent pivots.
  static constexpr int kFlooredOrder = 164;
  SmallEigen eig;
  SmallSolver(Runtime& r, int m_, double2* a, double2* b, double* w) : rt(r), m(m_) {
    const char* sel = std::getenv("HALF_SMALL_EIG");
    own = !(sel && std::string(sel) == "cusolver");
    if (const char* pr = std::getenv("HALF_PENCIL_RANGE")) range = std::string(pr) != "0";
    if (const char* po = std::getenv("HALF_PENCIL_OWN")) own_large = own && std::string(po) != "0";
    info.resize(3);
    info.zero(rt.stream);
    if (own) eig.reserve(rt, own_large ? 2 * m : std::min(2 * m, SmallEigen::kGridMaxOrder));   // locking shrinks pencils below it
    int l1 = 0, l2 = 0, l3 = 0;
    cusolver_check(cusolverDnZheevd_bufferSize(rt.solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, m,
                                               reinterpret_cast<cuDoubleComplex*>(a), m, w, &l1),
                   "zheevd buffer");
    cusolver_check(cusolverDnZhegvd_bufferSize(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                               CUBLAS_FILL_MODE_UPPER, 2 * m, reinterpret_cast<cuDoubleComplex*>(a),
                                               2 * m, reinterpret_cast<cuDoubleComplex*>(b), 2 * m, w, &l2),
                   "zhegvd buffer");
    cusolver_check(cusolverDnZhegvd_bufferSize(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                               CUBLAS_FILL_MODE_UPPER, m, reinterpret_cast<cuDoubleComplex*>(a), m,
                                               reinterpret_cast<cuDoubleComplex*>(b), m, w, &l3),
                   "zhegvd buffer");
    int l4 = 0, l5 = 0, meig = 0;
    cusolver_check(cusolverDnZhegvdx_bufferSize(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                                CUSOLVER_EIG_RANGE_I, CUBLAS_FILL_MODE_UPPER, 2 * m,
                                                reinterpret_cast<cuDoubleComplex*>(a), 2 * m,
                                                reinterpret_cast<cuDoubleComplex*>(b), 2 * m, 0.0, 0.0, 1, m, &meig, w,
                                                &l4),
                   "zhegvdx buffer");
    cusolver_check(cusolverDnZhegvdx_bufferSize(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                                CUSOLVER_EIG_RANGE_I, CUBLAS_FILL_MODE_UPPER, m,
                                                reinterpret_cast<cuDoubleComplex*>(a), m,
                                                reinterpret_cast<cuDoubleComplex*>(b), m, 0.0, 0.0, 1, m, &meig, w, &l5),
                   "zhegvdx buffer");
    work.resize(size_t(std::max({l1, l2, l3, l4, l5, 1})));
    lw_ev = l1;
    lw_gv = std::max(l2, l3);
  }
  // all n eigenpairs of a (n x n) (cuSOLVER in all modes: metrics above kFlooredOrder)
  void heevd(double2* a, int n, double* w) {
    cusolver_check(cusolverDnZheevd(rt.solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, n,
                                    reinterpret_cast<cuDoubleComplex*>(a), n, w,
                                    reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()), info.get()),
                   "zheevd");
  }
  // orders of the own solver; those of the grid-wide tridiagonalisation in the
  // guard-band modes only (the FP64 mode keeps zhegvd there)
  bool own_order(int n) const { return own_kernels(n) || (own && own_large); }
  // those of its own kernels, which scale the pencil themselves
  bool own_kernels(int n) const {
    return own && (SmallEigen::cluster_order(rt, n) || (range && SmallEigen::grid_order(rt, n)));
  }
  // generalized problem of order n; the nev lowest eigenvectors are wanted
  void hegvd(double2* a, double2* b, int n, double* w, int nev) {
    if (own_order(n)) {
      eig.hegv(rt, a, b, n, nev, w, info.get() + 1, info.get() + 2, n > kFlooredOrder);
      return;
    }
    if (range) {
      int meig = 0;   // the routine returns it through host memory (it synchronises the stream)
      cusolver_check(cusolverDnZhegvdx(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUSOLVER_EIG_RANGE_I,
                                       CUBLAS_FILL_MODE_UPPER, n, reinterpret_cast<cuDoubleComplex*>(a), n,
                                       reinterpret_cast<cuDoubleComplex*>(b), n, 0.0, 0.0, 1, nev, &meig, w,
                                       reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()),
                                       info.get() + 1),
                     "zhegvdx");
      return;
    }
    cusolver_check(cusolverDnZhegvd(rt.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER,
                                    n, reinterpret_cast<cuDoubleComplex*>(a), n, reinterpret_cast<cuDoubleComplex*>(b),
                                    n, w, reinterpret_cast<cuDoubleComplex*>(work.get()), int(work.size()),
                                    info.get() + 1),
                   "zhegvd");
  }
};

// Block state of one precision.
template <typename R>
struct Blocks {
  using C = cplx_t<R>;
  int n = 0, m = 0;
  DeviceBuffer<C> X[2], HX[2], SX[2];
  DeviceBuffer<C> P, HP, SP, PU, HPU, SPU;   // PU, HPU, SPU from the first metric step on
  DeviceBuffer<C> small;       // m x m (cross) in this precision
  DeviceBuffer<C> Y;           // 2m x m rotation in this precision
  int cur = 0;
  void allocate(int n_, int m_) {
    n = n_; m = m_;
    size_t nm = size_t(n) * m;
    for (int i = 0; i < 2; ++i) { X[i].resize(nm); HX[i].resize(nm); SX[i].resize(nm); }
    P.resize(nm); HP.resize(nm); SP.resize(nm);
    small.resize(size_t(m) * m);
    Y.resize(size_t(2) * m * m);
  }
  C* x() { return X[cur].get(); }
  C* hx() { return HX[cur].get(); }
  C* sx() { return SX[cur].get(); }
};

struct Scratch64 {
  DeviceBuffer<double2> metric, hsub, ssub;   // m x m, 2m x 2m, 2m x 2m
  DeviceBuffer<double> w, mu, norms, kinetic, jacobi, report;
  DeviceBuffer<int> idx, active, perm;
};

// FP32 blocks projected into an ((m + np) x (m + np), ld m + np) FP64 matrix:
// [0:m,0:m] = A^H B1, [0:m,m:] = A^H B2, [m:,m:] = P^H B2 (the upper triangle
// is what zhegvd reads); tensor-core products written straight into the FP64
// pencil, split-K partial sums reduced in FP64.
void project_upper(Runtime& rt, int n, int m, int np, const float2* x, const float2* p, const float2* bx,
                   const float2* bp, double2* out) {
  const int ld = m + np;
  gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, m, m, n, x, n, bx, n, out, ld);
  gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, m, np, n, x, n, bp, n, out + (long long)m * ld, ld);
  gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, np, np, n, p, n, bp, n, out + (long long)m * ld + m, ld);
}

template <typename R>
struct AccRun {
  using C = cplx_t<R>;
  Context& ctx;
  KOperatorSet& ks;
  Runtime& rt;
  Blocks<R>& blk;
  Scratch64& sc;
  SmallSolver& ss;
  DeviceBuffer<C>& tmp2m;      // 2m x 2m in this precision (projection staging)
  int n, m, chunk;
  int mcheck = m;              // bands whose residuals decide convergence (guard bands excluded)
  bool guarded = false;        // guard-band modes: may skip the separate metric normalisation
  int metric_fallbacks = 0;    // Jacobi-scaled pencils whose Cholesky failed (redone with the metric step)
  int unchecked = 0;           // P columns of a step whose pencil status has not been read yet (redo_if_failed), or 0
  int nl = 0;                  // hard-locked columns, at the front of X, H X, S X
  std::vector<double> wh;      // Ritz values (host copy, physical column order)
  std::vector<int> req;        // requested bands: physical columns of the mcheck lowest Ritz values
  long long op_cols = 0;
  Tracer* tr = nullptr;
  void mark(const char* s) { if (tr) tr->mark(s); }
  // FP64 phase of a mixed solve: the projections and the S-orthogonalisation
  // may run on the integer tensor cores.  They hold an operand in fixed point
  // relative to its rows' norms (zcrt.cu has the errors, which there are below
  // ZGEMM's).  The rotations never do: a row of [X P] holds X beside P entries
  // as small as the residuals, and near convergence Y is close to the
  // identity, where ZGEMM loses next to nothing.
  bool integer = false;

  // (timed by the sweep's events: no host synchronisation)
  void apply(const C* x, C* hx, C* sx, int nb) {
    apply_hs<R>(ctx, ks, x, n, nb, hx, sx, chunk);
    op_cols += nb;
  }

  // small FP64 matrices -> FP32
  void to_r(const double2* in, long long ldi, float2* out, long long ldo, int rows, int cols) {
    convert_block_kernel<double2, float2><<<ceil_div((long long)rows * cols, 256), 256, 0, rt.stream>>>(in, ldi, out, ldo,
                                                                                                     rows, cols);
    ++rt.prof.launches;
  }

  // Rayleigh-Ritz on the current X only (m x m)
  void rayleigh_ritz_x() {
    double2* hs = sc.hsub.get();
    double2* ssb = sc.ssub.get();
    int nx = blk.cur ^ 1;
    if constexpr (sizeof(R) == 8) {
      const ZBlock b[2] = {{blk.hx(), m}, {blk.sx(), m}};
      double2* const c[2] = {hs, ssb};
      zgram(rt, n, {blk.x(), m}, b, c, 2, m, true, zgram_route(rt.sms, n, m, m, integer));
      ss.hegvd(hs, ssb, m, sc.w.get(), m);
      const ZBlock z[3] = {{blk.x(), m}, {blk.hx(), m}, {blk.sx(), m}};
      double2* const out[3] = {blk.X[nx].get(), blk.HX[nx].get(), blk.SX[nx].get()};
      zupdate(rt, n, z, hs, m, out, m, 3, 1.0, 0.0, zupdate_route(rt.sms, n, m, m, false));
    } else {
      const auto one = cval<R>(1.0), zero = cval<R>(0.0);
      gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, m, m, n, blk.x(), n, blk.hx(), n, hs, m);
      gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, m, m, n, blk.x(), n, blk.sx(), n, ssb, m);
      ss.hegvd(hs, ssb, m, sc.w.get(), m);
      to_r(hs, m, blk.Y.get(), m, m, m);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, m, m, one, blk.x(), n, blk.Y.get(), m, zero, blk.X[nx].get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, m, m, one, blk.hx(), n, blk.Y.get(), m, zero, blk.HX[nx].get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, m, m, one, blk.sx(), n, blk.Y.get(), m, zero, blk.SX[nx].get(), n);
    }
    blk.cur = nx;
  }

  // residual norms of the current Ritz pairs; returns the max norm over the
  // requested bands, which are the mcheck lowest Ritz values (req, physical
  // column indices in ascending order of their values; host sync)
  double residuals(std::vector<double>& norms, int* infos) {
    launch_chained(m, 256, 0, rt.stream, residual_norm_kernel<C>,
        blk.hx(), blk.sx(), n, n, sc.w.get(), ss.info.get(), rt.tc_err.get(), sc.norms.get(), sc.report.get());
    ++rt.prof.launches;
    HALF_LAUNCH("residual norms");
    const size_t words = size_t(2) * m + 4;
    double* host = rt.pinned(words);
    HALF_CUDA(cudaMemcpyAsync(host, sc.report.get(), words * sizeof(double), cudaMemcpyDeviceToHost, rt.stream));
    HALF_CUDA(cudaStreamSynchronize(rt.stream));
    norms.assign(host, host + m);
    wh.assign(host + m, host + 2 * m);
    for (int i = 0; i < 3; ++i) infos[i] = int(host[2 * m + i]);
    if (host[2 * m + 3] != 0.0) tc_check(rt);   // raises
    rt.crt_pending = false;
    mark("residual");
    if (redo_if_failed(infos)) return residuals(norms, infos);
    const std::string failure = pencil_failure(infos);
    if (!failure.empty()) fail(kInternal, failure);
    order_requested();
    double mx = 0;
    for (int j : req) mx = std::max(mx, norms[j]);
    return mx;
  }

  // req from the host Ritz values wh: locked columns keep their values, so
  // the physical order is ascending only without locking; a stable sort keeps
  // it where it is
  void order_requested() {
    req.resize(m);
    for (int j = 0; j < m; ++j) req[j] = j;
    std::stable_sort(req.begin(), req.end(), [&](int a, int b) { return wh[a] < wh[b]; });
    req.resize(std::min(mcheck, m));
  }

  // A guard-band pencil of the own solver went ahead unchecked, and its overlap
  // turned out not to be positive definite (or the solve failed): the step is
  // redone from the blocks it started from, with the metric normalisation.
  bool redo_if_failed(const int* infos) {
    const int np = unchecked;
    unchecked = 0;
    if (np == 0 || (infos[1] == 0 && infos[2] == 0)) return false;
    ++metric_fallbacks;
    ss.info.zero(rt.stream);
    blk.cur ^= 1;
    rayleigh_ritz(np, false);
    return true;
  }

  // After an iteration that no residual check followed (the iteration bound was reached).
  void settle() {
    if (unchecked == 0) return;
    int infos[3];
    HALF_CUDA(cudaMemcpyAsync(infos, ss.info.get(), sizeof infos, cudaMemcpyDeviceToHost, rt.stream));
    HALF_CUDA(cudaStreamSynchronize(rt.stream));
    redo_if_failed(infos);
  }

  // the current Ritz values to the host and req from them (as settle)
  void refresh_values() {
    settle();
    wh.resize(m);
    HALF_CUDA(cudaMemcpyAsync(wh.data(), sc.w.get(), m * sizeof(double), cudaMemcpyDeviceToHost, rt.stream));
    HALF_CUDA(cudaStreamSynchronize(rt.stream));
    order_requested();
  }

  // Hard locking: move the (unlocked) columns `newly` to the locked front
  // [0, nl) of X, H X, S X, of the Ritz values and of the host norms; locked
  // columns are no longer rotated or projected (their residuals stay as they
  // were), and P stays S-orthogonal to them through the orthogonalisation
  // against the whole of X.
  void lock(const std::vector<int>& newly, std::vector<double>& norms) {
    if (newly.empty()) return;
    std::vector<char> is_new(m, 0);
    for (int j : newly) is_new[j] = 1;
    std::vector<int> perm;
    perm.reserve(m);
    for (int j = 0; j < nl; ++j) perm.push_back(j);
    for (int j = nl; j < m; ++j)
      if (is_new[j]) perm.push_back(j);
    for (int j = nl; j < m; ++j)
      if (!is_new[j]) perm.push_back(j);
    sc.perm.upload(perm, rt.stream);
    const int nx = blk.cur ^ 1;
    const long long cnt = (long long)n * m;
    launch_chained(ceil_div(cnt, 256), 256, 0, rt.stream, gather_columns_kernel<C>,
        blk.x(), blk.X[nx].get(), n, m, sc.perm.get());
    launch_chained(ceil_div(cnt, 256), 256, 0, rt.stream, gather_columns_kernel<C>,
        blk.hx(), blk.HX[nx].get(), n, m, sc.perm.get());
    launch_chained(ceil_div(cnt, 256), 256, 0, rt.stream, gather_columns_kernel<C>,
        blk.sx(), blk.SX[nx].get(), n, m, sc.perm.get());
    launch_chained(ceil_div(m, 256), 256, 0, rt.stream, gather_values_kernel,
        sc.w.get(), sc.mu.get(), m, sc.perm.get());
    HALF_CUDA(cudaMemcpyAsync(sc.w.get(), sc.mu.get(), m * sizeof(double), cudaMemcpyDeviceToDevice, rt.stream));
    launch_chained(ceil_div(m, 256), 256, 0, rt.stream, gather_values_kernel,
        sc.norms.get(), sc.mu.get(), m, sc.perm.get());
    HALF_CUDA(cudaMemcpyAsync(sc.norms.get(), sc.mu.get(), m * sizeof(double), cudaMemcpyDeviceToDevice, rt.stream));
    HALF_LAUNCH("lock columns");
    rt.prof.launches += 5;
    blk.cur = nx;
    std::vector<double> nn(m), ww(m);
    for (int j = 0; j < m; ++j) {
      nn[j] = norms[perm[j]];
      ww[j] = wh[perm[j]];
    }
    norms.swap(nn);
    wh.swap(ww);
    nl += int(newly.size());
  }

  // one ACC iteration after the residual check (src/half_cuda_iterative_solver.cuf:158-195).
  // active (guard-band modes only; null = every band, the reference's step):
  // the bands whose correction directions enter P, in order.
  void iterate(double seed_threshold, const std::vector<int>* active = nullptr) {
    const auto one = cval<R>(1.0), zero = cval<R>(0.0), mone = cval<R>(-1.0);
    const int np = active ? int(active->size()) : m;
    const int* cols = nullptr;
    if (np < m) {
      sc.active.upload(*active, rt.stream);
      cols = sc.active.get();
    }
    long long nm = (long long)n * np;
    launch_chained(ceil_div(nm, 256), 256, 0, rt.stream, precondition_kernel<C>,
        blk.hx(), blk.sx(), n, n, m, np, cols, sc.w.get(), sc.norms.get(), seed_threshold, sc.kinetic.get(),
        blk.P.get());
    ++rt.prof.launches;
    HALF_LAUNCH("precondition");
    mark("precondition");
    apply(blk.P.get(), blk.HP.get(), blk.SP.get(), np);
    mark("apply");
    // S-orthogonalise against X
    if constexpr (sizeof(R) == 8) {
      const ZBlock b = {blk.SP.get(), np};
      double2* const c = blk.small.get();
      zgram(rt, n, {blk.x(), m}, &b, &c, 1, m, false, zgram_route(rt.sms, n, m, np, integer));
      const ZBlock z[3] = {{blk.x(), m}, {blk.hx(), m}, {blk.sx(), m}};
      double2* const out[3] = {blk.P.get(), blk.HP.get(), blk.SP.get()};
      zupdate(rt, n, z, blk.small.get(), m, out, np, 3, -1.0, 1.0, zupdate_route(rt.sms, n, m, np, integer));
    } else {
      gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, m, np, n, one, blk.x(), n, blk.SP.get(), n, zero, blk.small.get(), m);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, m, mone, blk.x(), n, blk.small.get(), m, one, blk.P.get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, m, mone, blk.hx(), n, blk.small.get(), m, one, blk.HP.get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, m, mone, blk.sx(), n, blk.small.get(), m, one, blk.SP.get(), n);
    }
    mark("orth_gemm");
    rayleigh_ritz(np, guarded && ss.own);
  }

  // The rest of the iteration, from P, HP, SP (np columns, S-orthogonal to X):
  // metric normalisation unless skipped, Rayleigh-Ritz, rotation.
  void rayleigh_ritz(int np, bool skip_metric) {
    const auto one = cval<R>(1.0), zero = cval<R>(0.0);
    // In the guard-band modes the separate S-metric normalisation is
    // skipped.  The pencil is Jacobi-scaled (the library's own kernels do that
    // themselves) and goes through a plain Cholesky of the overlap, which does
    // the metric step's work; if that Cholesky (or the solve) fails, the step
    // is redone with the metric normalisation.  The own kernels' status is read
    // with the next residuals, the others' here.  To order 164 the own solver
    // floors dependent pivots exactly like the metric step instead, so [X P]
    // spans the same space and the Ritz pairs are the same.  (Floored pivots at
    // larger orders let rounding in the FP32 phase's overlaps through as Ritz
    // values of -1e9 eV: 600 bands of the 12-atom cell.)  The FP64 mode keeps
    // the reference's metric step.
    // Rayleigh-Ritz on Z = [X_U PU], X_U = the unlocked columns [nl, m) of X
    // (all of them without hard locking)
    const int mu = m - nl;
    const long long off = (long long)nl * n;
    const int ord = mu + np;
    const bool own_pencil = ss.own_kernels(ord);
    unchecked = skip_metric && own_pencil && ord > SmallSolver::kFlooredOrder ? np : 0;
    double2* hs = sc.hsub.get();
    double2* ssb = sc.ssub.get();
    double* wu = sc.w.get() + nl;
    C* pu = blk.P.get();
    C* hpu = blk.HP.get();
    C* spu = blk.SP.get();
    auto use_metric = [&]() {
      normalise_metric(one, zero, np);
      pu = blk.PU.get();
      hpu = blk.HPU.get();
      spu = blk.SPU.get();
    };
    if (!skip_metric) use_metric();
    auto project = [&]() {
      if constexpr (sizeof(R) == 8) {
        const ZBlock b[2] = {{blk.hx() + off, mu, hpu, np}, {blk.sx() + off, mu, spu, np}};
        double2* const c[2] = {hs, ssb};
        zgram(rt, n, {blk.x() + off, mu, pu, np}, b, c, 2, ord, true, zgram_route(rt.sms, n, ord, ord, integer));
      } else {
        project_upper(rt, n, mu, np, blk.x() + off, pu, blk.hx() + off, hpu, hs);
        project_upper(rt, n, mu, np, blk.x() + off, pu, blk.sx() + off, spu, ssb);
      }
    };
    project();
    mark("rr_gemm");
    if (skip_metric && !own_pencil) {
      jacobi_diag_kernel<<<ceil_div(ord, 256), 256, 0, rt.stream>>>(ssb, ord, sc.jacobi.get());
      jacobi_scale_kernel<<<ceil_div((long long)ord * ord, 256), 256, 0, rt.stream>>>(hs, ssb, ord, sc.jacobi.get());
      HALF_LAUNCH("Jacobi scaling");
      rt.prof.launches += 2;
      ss.hegvd(hs, ssb, ord, wu, mu);
      int st[2] = {0, 0};   // solve status, Cholesky status (own solver)
      HALF_CUDA(cudaMemcpyAsync(st, ss.info.get() + 1, 2 * sizeof(int), cudaMemcpyDeviceToHost, rt.stream));
      HALF_CUDA(cudaStreamSynchronize(rt.stream));
      if (st[0] == 0 && st[1] == 0) {
        scale_rows_kernel<<<ceil_div((long long)ord * mu, 256), 256, 0, rt.stream>>>(hs, ord, ord, mu, sc.jacobi.get());
        ++rt.prof.launches;
      } else {
        ++metric_fallbacks;
        use_metric();
        project();
        ss.hegvd(hs, ssb, ord, wu, mu);
      }
    } else {
      ss.hegvd(hs, ssb, ord, wu, mu);
    }
    mark("hegvd");
    int nx = blk.cur ^ 1;
    if constexpr (sizeof(R) == 8) {
      const ZBlock z[3] = {{blk.x() + off, mu, pu, np}, {blk.hx() + off, mu, hpu, np}, {blk.sx() + off, mu, spu, np}};
      double2* const out[3] = {blk.X[nx].get() + off, blk.HX[nx].get() + off, blk.SX[nx].get() + off};
      zupdate(rt, n, z, hs, ord, out, mu, 3, 1.0, 0.0, zupdate_route(rt.sms, n, ord, mu, false));
    } else {
      rotate(ord, mu, np, off, pu, hpu, spu, hs, nx);
    }
    if (nl > 0) {   // locked columns go along unchanged
      const size_t bytes = size_t(off) * sizeof(C);
      HALF_CUDA(cudaMemcpyAsync(blk.X[nx].get(), blk.x(), bytes, cudaMemcpyDeviceToDevice, rt.stream));
      HALF_CUDA(cudaMemcpyAsync(blk.HX[nx].get(), blk.hx(), bytes, cudaMemcpyDeviceToDevice, rt.stream));
      HALF_CUDA(cudaMemcpyAsync(blk.SX[nx].get(), blk.sx(), bytes, cudaMemcpyDeviceToDevice, rt.stream));
    }
    blk.cur = nx;
    mark("rr_rot");
  }

  // FP32: X[nx], HX[nx], SX[nx] from column offset off on = [X_U pu] Y and the same of H and S, Y = hs (ord x mu, FP64)
  void rotate(int ord, int mu, int np, long long off, const C* pu, const C* hpu, const C* spu, const double2* hs,
              int nx) {
    const auto one = cval<R>(1.0), zero = cval<R>(0.0);
    to_r(hs, ord, blk.Y.get(), ord, ord, mu);
    const C* ytop = blk.Y.get();
    const C* ybot = blk.Y.get() + mu;
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, mu, one, blk.x() + off, n, ytop, ord, zero, blk.X[nx].get() + off, n);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, np, one, pu, n, ybot, ord, one, blk.X[nx].get() + off, n);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, mu, one, blk.hx() + off, n, ytop, ord, zero, blk.HX[nx].get() + off, n);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, np, one, hpu, n, ybot, ord, one, blk.HX[nx].get() + off, n);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, mu, one, blk.sx() + off, n, ytop, ord, zero, blk.SX[nx].get() + off, n);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, mu, np, one, spu, n, ybot, ord, one, blk.SX[nx].get() + off, n);
  }

  // S-metric normalisation of the np columns of P, HP, SP into PU, HPU, SPU
  // (src/half_cuda_iterative_solver.cuf:166-176)
  void normalise_metric(cplx_t<R> one, cplx_t<R> zero, int np) {
    double2* metric = sc.metric.get();
    for (auto* b : {&blk.PU, &blk.HPU, &blk.SPU}) b->resize(size_t(n) * m);
    if constexpr (sizeof(R) == 8) {
      const ZBlock b = {blk.SP.get(), np};
      zgram(rt, n, {blk.P.get(), np}, &b, &metric, 1, np, true, zgram_route(rt.sms, n, np, np, integer));
    } else {
      gemm_to64(rt, CUBLAS_OP_C, CUBLAS_OP_N, np, np, n, blk.P.get(), n, blk.SP.get(), n, metric, np);
    }
    mark("metric_gemm");
    // Above order 164 the reference's eigenvectors with its absolute floor: late
    // in a solve P is so small that rounding in the metric lies far below that
    // floor, while the Cholesky factor's, relative to the scaled diagonal, lies
    // in it, and the step that is redone for an indefinite overlap (rayleigh_ritz)
    // must not meet one again.
    if (!(ss.own && np <= SmallSolver::kFlooredOrder && ss.eig.metric_normalize(rt, metric, np, ss.info.get()))) {
      ss.heevd(metric, np, sc.mu.get());
      scale_columns_kernel<<<ceil_div(np * np, 256), 256, 0, rt.stream>>>(metric, np, sc.mu.get(), 1.0e-14);
      ++rt.prof.launches;
    }
    mark("heevd");
    if constexpr (sizeof(R) == 8) {
      const ZBlock z[3] = {{blk.P.get(), np}, {blk.HP.get(), np}, {blk.SP.get(), np}};
      double2* const out[3] = {blk.PU.get(), blk.HPU.get(), blk.SPU.get()};
      zupdate(rt, n, z, metric, np, out, np, 3, 1.0, 0.0, zupdate_route(rt.sms, n, np, np, false));
    } else {
      to_r(metric, np, blk.small.get(), np, np, np);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, np, one, blk.P.get(), n, blk.small.get(), np, zero, blk.PU.get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, np, one, blk.HP.get(), n, blk.small.get(), np, zero, blk.HPU.get(), n);
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, np, np, one, blk.SP.get(), n, blk.small.get(), np, zero, blk.SPU.get(), n);
    }
    mark("metric_rot");
  }
};

}  // namespace

void solve_acc(Context& ctx, KOperatorSet& ks, int nbands, bool want_vectors, SolveOutput& out, SolveInfo& info) {
  auto t_start = std::chrono::steady_clock::now();
  Runtime& rt = *ks.rt;
  const int n = int(ks.basis.npw());
  const int mreq = nbands;
  if (mreq < 1 || mreq > n) fail(kInvalidArgument, "invalid ACC target band count");
  if (2 * mreq > n) fail(kInvalidArgument, "ACC solver requires NBANDS <= NPL/2");
  const AccControls& cfg = ctx.acc;
  const bool mixed = cfg.precision == kMixed;
  // The mixed and guarded modes carry guard bands (m/4, at least 4, within
  // NPL/2): a requested edge band nearly degenerate with the first
  // unrequested one otherwise converges at the block method's edge rate
  // (after the FP32 phase up to ten times the FP64 iteration count), and a
  // degenerate level cut by the band count can leave the block converged on
  // a higher level.  Convergence is decided on the requested bands only; the
  // FP64 mode is the reference algorithm unchanged (no guard bands).
  const bool guarded = mixed || cfg.precision == kFP64Guarded;
  // m / 4 guard bands: on the 216-atom cell with hard locking, m/8, m/5, m/4,
  // m/3 and m/2 gave 48, 31, 25, 22 and 17 iterations and 1.34, 1.18, 1.15,
  // 1.19 and 1.23 s per k point (the extra columns cost more than the
  // iterations they save beyond m/4).  HALF_GUARD_DIV overrides the divisor.
  int guard_div = 4;
  if (const char* gd = std::getenv("HALF_GUARD_DIV")) guard_div = std::max(1, std::atoi(gd));
  const int guard = guarded ? std::min(std::max(4, mreq / guard_div), n / 2 - mreq) : 0;
  const int m = mreq + guard;
  Scratch64 sc;
  sc.metric.resize(size_t(m) * m);
  sc.hsub.resize(size_t(4) * m * m);
  sc.ssub.resize(size_t(4) * m * m);
  sc.w.resize(2 * m);
  sc.jacobi.resize(2 * m);
  sc.mu.resize(m);
  sc.norms.resize(m);
  sc.report.resize(2 * size_t(m) + 4);
  sc.kinetic.upload(ks.basis.kinetic, rt.stream);
  auto order = kinetic_order(ks.basis.kinetic);
  order.resize(m);
  sc.idx.upload(order, rt.stream);
  SmallSolver ss(rt, m, sc.hsub.get(), sc.ssub.get(), sc.w.get());
  ss.range = ss.range && guarded;   // the FP64 mode keeps the reference's zhegvd
  const double seed_threshold = std::max(cfg.tol * 1e-2, 1e-12);
  std::vector<double> norms;
  // Soft locking (guard-band modes): a requested band whose residual is at or
  // below half the phase's tolerance keeps its Ritz vector in X but adds no
  // correction direction to P, so late iterations solve pencils of order
  // m + (active bands) instead of 2m and apply the operator to fewer columns.
  // The set is recomputed every iteration (a band whose residual rises is
  // active again); guard bands are always active.  On by default in the
  // guard-band modes (on the 216-atom cell it cut the mixed solve from 3.8 s
  // to 2.2 s per k point); environment HALF_SOFT_LOCK=0 turns it off, and the
  // FP64 mode, the reference's iteration, never locks.
  bool soft_lock = guarded;
  if (const char* sl = std::getenv("HALF_SOFT_LOCK")) soft_lock = guarded && std::string(sl) != "0";
  // Hard locking (on with soft locking; HALF_HARD_LOCK=0 keeps the soft
  // variant): a requested band at or below the lock tolerance leaves the
  // iteration for the rest of the phase.  Its column moves to the locked
  // front of X, H X, S X and is neither projected nor rotated again, so the
  // pencils have order 2 (m - locked) and the rotations and projections
  // shrink with them; P is still S-orthogonalised against the whole of X.
  // On the 216-atom cell 235-470 of the 480 requested bands sit at or below
  // the lock tolerance in most iterations of both phases.  Locks are
  // released when the FP32 phase hands over to FP64.
  // lock tolerance = lock_frac x the phase's tolerance (HALF_LOCK_FRACTION
  // overrides 0.5: measurement runs)
  double lock_frac = 0.5;
  if (const char* lf = std::getenv("HALF_LOCK_FRACTION")) lock_frac = std::min(1.0, std::max(0.0, std::atof(lf)));
  bool hard_lock = soft_lock;
  if (const char* hl = std::getenv("HALF_HARD_LOCK")) hard_lock = soft_lock && std::string(hl) != "0";
  std::vector<int> active;
  auto pick_active = [&](double lock_tol) -> const std::vector<int>* {
    if (!soft_lock) return nullptr;
    active.clear();
    for (int j = 0; j < m; ++j)
      if (j >= mreq || !(norms[j] <= lock_tol)) active.push_back(j);
    return &active;
  };
  // one iteration of a phase: hard-lock the newly converged requested bands
  // and iterate on the rest, or the soft-locked / reference step
  auto advance = [&](auto& run, double lock_tol) {
    if (!hard_lock) {
      run.iterate(seed_threshold, pick_active(lock_tol));
      return;
    }
    std::vector<int> newly;
    for (int j : run.req)
      if (j >= run.nl && norms[j] <= lock_tol && run.nl + int(newly.size()) + 1 < m) newly.push_back(j);
    std::sort(newly.begin(), newly.end());
    run.lock(newly, norms);
    active.clear();
    for (int j = run.nl; j < m; ++j) active.push_back(j);
    run.iterate(seed_threshold, &active);
  };
  int infos[3] = {0, 0, 0};
  int iter = 0, fp64_iter = 0;
  bool converged = false;
  double max_res = HUGE_VAL;
  long long op_cols = 0;

  int fallbacks = 0;
  Blocks<double> b64;
  b64.allocate(n, m);
  DeviceBuffer<double2> tmp64(size_t(4) * m * m);
  Tracer tracer;
  tracer.s = rt.stream;
  AccRun<double> run64{ctx, ks, rt, b64, sc, ss, tmp64, n, m, cfg.block};
  run64.tr = &tracer;
  run64.mcheck = mreq;
  run64.guarded = guarded;
  run64.integer = mixed;

  if (mixed) {
    // ---------------- FP32 phase
    Blocks<float> b32;
    b32.allocate(n, m);
    DeviceBuffer<float2> tmp32(size_t(4) * m * m);
    AccRun<float> run32{ctx, ks, rt, b32, sc, ss, tmp32, n, m, cfg.block};
    run32.tr = &tracer;
    run32.mcheck = mreq;
    run32.guarded = guarded;
    init_states_kernel<float2><<<ceil_div((long long)n * m, 256), 256, 0, rt.stream>>>(b32.x(), n, n, m, sc.idx.get());
    ++rt.prof.launches;
    run32.apply(b32.x(), b32.hx(), b32.sx(), m);
    run32.rayleigh_ritz_x();
    // Switch to FP64 once the residual is in the FP32 regime or stops improving.
    // (HALF_FP32_SWITCH_EV overrides the 3e-3 eV switch point: measurement runs)
    double switch_ev = 3.0e-3;
    if (const char* sw = std::getenv("HALF_FP32_SWITCH_EV")) switch_ev = std::max(1e-8, std::atof(sw));
    const double switch_tol = std::max(cfg.tol, switch_ev);
    double best = HUGE_VAL;
    int since_best = 0;
    for (iter = 1; iter <= cfg.max_iter; ++iter) {
      max_res = run32.residuals(norms, infos);
      tracer.step("fp32", iter, max_res, norms, mreq, lock_frac * switch_tol);
      if (max_res < 0.9 * best) { best = max_res; since_best = 0; } else { ++since_best; }
      if (max_res <= switch_tol || since_best >= 6) break;
      advance(run32, lock_frac * switch_tol);
    }
    if (iter > cfg.max_iter) iter = cfg.max_iter;
    run32.settle();
    op_cols += run32.op_cols;
    fallbacks += run32.metric_fallbacks;
    // promote X, recreate H X and S X in FP64, Rayleigh-Ritz
    convert_kernel<float2, double2><<<ceil_div((long long)n * m, 256), 256, 0, rt.stream>>>(b32.x(), b64.x(), (long long)n * m);
    ++rt.prof.launches;
    run64.apply(b64.x(), b64.hx(), b64.sx(), m);
    run64.rayleigh_ritz_x();
    for (fp64_iter = 1; fp64_iter <= cfg.max_iter; ++fp64_iter) {
      max_res = run64.residuals(norms, infos);
      tracer.step("fp64", fp64_iter, max_res, norms, mreq, lock_frac * cfg.tol);
      if (max_res <= cfg.tol) { converged = true; break; }
      advance(run64, lock_frac * cfg.tol);
    }
    fp64_iter = std::min(fp64_iter, cfg.max_iter);
    iter += fp64_iter;
  } else {
    init_states_kernel<double2><<<ceil_div((long long)n * m, 256), 256, 0, rt.stream>>>(b64.x(), n, n, m, sc.idx.get());
    ++rt.prof.launches;
    run64.apply(b64.x(), b64.hx(), b64.sx(), m);
    run64.rayleigh_ritz_x();
    for (iter = 1; iter <= cfg.max_iter; ++iter) {
      max_res = run64.residuals(norms, infos);
      tracer.step("fp64", iter, max_res, norms, mreq, lock_frac * cfg.tol);
      if (max_res <= cfg.tol) { converged = true; break; }
      advance(run64, lock_frac * cfg.tol);
    }
    iter = std::min(iter, cfg.max_iter);
    fp64_iter = iter;
  }
  op_cols += run64.op_cols;
  fallbacks += run64.metric_fallbacks;
  // the requested eigenpairs in ascending order (req: physical columns, from
  // the last residual check; the identity order unless bands were locked)
  if (!converged) run64.refresh_values();   // the last step was an iteration, not a residual check
  const std::vector<int>& req = run64.req;
  if (int(req.size()) != mreq) fail(kInternal, "ACC finished without Ritz values");
  out.eigenvalues.resize(mreq);
  for (int i = 0; i < mreq; ++i) out.eigenvalues[i] = run64.wh[req[i]];
  out.overlap_min = -1.0;   // src/half_cuda_iterative_solver.cuf:200
  out.overlap_max = -1.0;
  out.dvectors.resize(size_t(n) * mreq);
  sc.perm.upload(req, rt.stream);
  launch_chained(ceil_div((long long)n * mreq, 256), 256, 0, rt.stream, gather_columns_kernel<double2>,
      b64.x(), out.dvectors.get(), n, mreq, sc.perm.get());
  HALF_LAUNCH("ACC output gather");
  ++rt.prof.launches;
  if (want_vectors) {
    out.vectors.resize(size_t(2) * n * mreq);
    HALF_CUDA(cudaMemcpyAsync(out.vectors.data(), out.dvectors.get(), size_t(n) * mreq * sizeof(double2),
                              cudaMemcpyDeviceToHost, rt.stream));
  }
  HALF_CUDA(cudaStreamSynchronize(rt.stream));
  tracer.report(iter);
  if (tracer.on && fallbacks) std::fprintf(stderr, "HALF Jacobi-scaled pencils redone with the metric step: %d\n", fallbacks);
  info.iterations = iter;
  info.fp64_iterations = fp64_iter;
  info.converged = converged ? 1 : 0;
  info.max_residual = max_res;
  info.npw = n;
  info.operator_columns = op_cols;
  info.solve_ms = ms_since(t_start);
  if (!converged && max_res > std::max(100.0 * cfg.tol, 1e-2))
    std::fprintf(stderr, "HALF ACC warning: stopped after %d iterations; max residual=%12.4E\n", cfg.max_iter, max_res);
}

}  // namespace hb
