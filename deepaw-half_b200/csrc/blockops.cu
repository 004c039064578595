// FP64 products of the acc iteration's band blocks (see blockops.h).
//
// An iteration of the FP64 phase projects [X P] against H and S of it,
// S-orthogonalises P, HP and SP against X, and rotates three blocks.  As
// separate ZGEMM calls those are 15 products (six projections, each with a
// split-K reduction, four of the orthogonalisation, six rotations), and on
// the small cells each is a launch or two of 5-10 us that leaves most of the
// GPU idle.  Here the projections are one launch plus one ordered reduction,
// the orthogonalisation two and the rotations one: [X P] is read as one block,
// the pencil's two matrices share the launch, tiles below the diagonal are
// skipped, and split-K fills the GPU.  On the 2-atom cell's FP64 iteration
// (16 bands, 725 plane waves, B200) the products took 133 us in 27 launches
// and take 53 us in 9.
//
// Both kernels are register-tiled FP64 FMA (4 x 4 complex accumulators per
// thread; 64 FMAs per 8 shared-memory loads), fed by cp.async two chunks deep.
// On the FP64 pipe they are about as fast as cuBLAS's DMMA kernels (the B200's
// FP64 vector and tensor rates are alike) but not faster, so products that
// fill the GPU by themselves go to cuBLAS or, in the FP64 phase of a mixed
// solve, to the integer tensor cores (zcrt.cu).
#include <algorithm>

#include "blas.h"
#include "blockops.h"
#include "zcrt.h"

namespace hb {

namespace {

__device__ __forceinline__ void copy16_or_zero(void* dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(on ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ const double2* column(const ZBlock& b, int j, int n) {
  return j < b.c1 ? b.p1 + (long long)j * n : b.p2 + (long long)(j - b.c1) * n;
}

__device__ __forceinline__ void fma_conj(double2& c, double2 a, double2 b) {   // c += conj(a) b
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(-a.y, b.x, c.y);
}
__device__ __forceinline__ void fma_plain(double2& c, double2 a, double2 b) {   // c += a b
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
}

constexpr int kT = 32;            // tile of the Gram kernel, and columns of the update kernel's
constexpr int kGramK = 32;        // rows of the blocks per chunk
constexpr int kGramPitch = kGramK + 1;
constexpr int kGramThreads = 64;
constexpr size_t kGramSmem = size_t(2) * 2 * kT * kGramPitch * sizeof(double2);

struct GramArgs {
  ZBlock a, b[2];
  double2* c[2];
  int n, ldc, rows, cols;
  int tiles_i, tiles_j, tiles;   // tiles per product (upper: those with i <= j)
  bool upper;
};

__device__ __forceinline__ void gram_tile(const GramArgs& g, int t, int& p, int& ti, int& tj) {
  p = t >= g.tiles;
  t -= p * g.tiles;
  if (!g.upper) {
    tj = t / g.tiles_i;
    ti = t - tj * g.tiles_i;
    return;
  }
  tj = 0;
  while (t > tj) {   // column tj of the upper triangle holds tj + 1 tiles
    t -= tj + 1;
    ++tj;
  }
  ti = t;
}

// One CTA per (tile, slice of kper rows): 64 threads, thread (ti, tj) owns
// rows ti + 8 r and columns tj + 8 q of the 32 x 32 tile.
__global__ void __launch_bounds__(kGramThreads) zgram_kernel(GramArgs g, int kper, int slices,
                                                             double2* __restrict__ partial) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* const sa = reinterpret_cast<double2*>(smem_raw);   // [2][kT][kGramPitch]
  double2* const sb = sa + 2 * kT * kGramPitch;
  int p, bi, bj;
  gram_tile(g, blockIdx.x, p, bi, bj);
  const ZBlock& B = g.b[p];
  const int i0 = bi * kT, j0 = bj * kT, n = g.n;
  const int k0 = blockIdx.y * kper, k1 = min(n, k0 + kper);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto load = [&](int buf, int k) {
    const int row = k + lane;
    const bool in = row < k1;
#pragma unroll 4
    for (int c = warp; c < kT; c += 2) {
      const bool ain = in && i0 + c < g.rows, bin = in && j0 + c < g.cols;
      copy16_or_zero(sa + (buf * kT + c) * kGramPitch + lane, ain ? column(g.a, i0 + c, n) + row : g.a.p1, ain);
      copy16_or_zero(sb + (buf * kT + c) * kGramPitch + lane, bin ? column(B, j0 + c, n) + row : B.p1, bin);
    }
    copies_commit();
  };
  double2 acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[r][q] = make_double2(0.0, 0.0);
  const int ti = tid & 7, tj = tid >> 3;
  int buf = 0;
  load(0, k0);
  for (int k = k0; k < k1; k += kGramK, buf ^= 1) {
    if (k + kGramK < k1) {
      load(buf ^ 1, k + kGramK);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    const double2* a = sa + (buf * kT + ti) * kGramPitch;
    const double2* b = sb + (buf * kT + tj) * kGramPitch;
#pragma unroll 4
    for (int kk = 0; kk < kGramK; ++kk) {
      double2 av[4], bv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        av[r] = a[8 * r * kGramPitch + kk];
        bv[r] = b[8 * r * kGramPitch + kk];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) fma_conj(acc[r][q], av[r], bv[q]);
    }
    __syncthreads();
  }
  if (slices == 1) {
    double2* c = g.c[p];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = i0 + ti + 8 * r, j = j0 + tj + 8 * q;
        if (i < g.rows && j < g.cols) c[(long long)j * g.ldc + i] = acc[r][q];
      }
    return;
  }
  double2* w = partial + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * (kT * kT);
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) w[(tj + 8 * q) * kT + ti + 8 * r] = acc[r][q];
}

// C = the slices' tiles added in order; one CTA of 256 threads per quarter tile.
__global__ void __launch_bounds__(256) zgram_reduce_kernel(GramArgs g, int slices, const double2* __restrict__ partial) {
  after_previous();
  const int tile = blockIdx.x >> 2, e = (blockIdx.x & 3) * 256 + threadIdx.x, tiles = gridDim.x >> 2;
  int p, bi, bj;
  gram_tile(g, tile, p, bi, bj);
  const int i = bi * kT + (e & 31), j = bj * kT + (e >> 5);
  if (i >= g.rows || j >= g.cols) return;
  double2 s = make_double2(0.0, 0.0);
  for (int z = 0; z < slices; ++z) s = cadd(s, partial[((long long)z * tiles + tile) * (kT * kT) + e]);
  g.c[p][(long long)j * g.ldc + i] = s;
}

constexpr int kUpRows = 64, kUpK = 16, kUpThreads = 128, kUpPitch = kUpK + 1;
constexpr size_t kUpSmem = size_t(2) * (kUpK * kUpRows + kT * kUpPitch) * sizeof(double2);

struct UpdateArgs {
  ZBlock z[3];
  double2* c[3];
  const double2* y;
  int n, ldy, cols;
  double alpha, beta;
};

// One CTA per (64 rows, 32 columns, block): 128 threads, thread (ti, tj) owns
// rows ti + 16 r and columns tj + 8 q.
__global__ void __launch_bounds__(kUpThreads) zupdate_kernel(UpdateArgs u) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* const sz = reinterpret_cast<double2*>(smem_raw);   // [2][kUpK][kUpRows]
  double2* const sy = sz + 2 * kUpK * kUpRows;                // [2][kT][kUpPitch]
  const ZBlock& Z = u.z[blockIdx.z];
  const int K = Z.c1 + Z.c2, n = u.n;
  const int r0 = blockIdx.x * kUpRows, j0 = blockIdx.y * kT;
  const int tid = threadIdx.x;
  auto load = [&](int buf, int k) {
    const int row = r0 + (tid & 63);
#pragma unroll
    for (int q = 0; q < kUpK / 2; ++q) {
      const int kl = (tid >> 6) + 2 * q;
      const bool on = row < n && k + kl < K;
      copy16_or_zero(sz + (buf * kUpK + kl) * kUpRows + (tid & 63), on ? column(Z, k + kl, n) + row : u.y, on);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int kl = tid & 15, c = (tid >> 4) + 8 * q;
      const bool on = k + kl < K && j0 + c < u.cols;
      copy16_or_zero(sy + (buf * kT + c) * kUpPitch + kl, on ? u.y + (long long)(j0 + c) * u.ldy + k + kl : u.y, on);
    }
    copies_commit();
  };
  double2 acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[r][q] = make_double2(0.0, 0.0);
  const int ti = tid & 15, tj = tid >> 4;
  int buf = 0;
  load(0, 0);
  for (int k = 0; k < K; k += kUpK, buf ^= 1) {
    if (k + kUpK < K) {
      load(buf ^ 1, k + kUpK);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    const double2* a = sz + buf * kUpK * kUpRows + ti;
    const double2* b = sy + (buf * kT + tj) * kUpPitch;
#pragma unroll 4
    for (int kk = 0; kk < kUpK; ++kk) {
      double2 av[4], bv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        av[r] = a[kk * kUpRows + 16 * r];
        bv[r] = b[8 * r * kUpPitch + kk];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) fma_plain(acc[r][q], av[r], bv[q]);
    }
    __syncthreads();
  }
  double2* const C = u.c[blockIdx.z];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = j0 + tj + 8 * q;
    if (j >= u.cols) break;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = r0 + ti + 16 * r;
      if (row < n) {
        double2* c = C + (long long)j * n + row;
        double2 v = cscale(acc[r][q], u.alpha);
        if (u.beta != 0.0) v = cadd(v, *c);
        *c = v;
      }
    }
  }
}

}  // namespace

namespace {

// The line lies where the fused kernels' time meets cuBLAS's, measured on whole
// FP64 solves (cuBLAS / fused, ms): 2-atom cell, order 32: 144 / 133; 12-atom
// cell, orders 80, 160 and 300: 16.8 / 14.8, 19.8 / 19.3, 31.3 / 32.3; 64-atom
// cell, orders 150 and 400: 60.5 / 60.6, 121 / 135.
bool zblock_small(int n, int order) { return double(n) * order * order < 2.0e8; }

CrtSide side_of(const ZBlock& b, int n, bool k_is_rows, bool conj) {
  CrtSide s;
  s.p = b.p1;
  s.p2 = b.p2;
  s.split = b.c2 > 0 ? b.c1 : INT32_MAX;
  s.ld = n;
  s.rows = k_is_rows ? b.cols() : n;
  s.k = k_is_rows ? n : b.cols();
  s.kcontig = k_is_rows;
  s.conj = conj;
  return s;
}

}  // namespace

ZRoute zgram_route(int sms, int n, int rows, int cols, bool integer) {
  if (zblock_small(n, std::max(rows, cols))) return ZRoute::kBlock;
  return integer && zcrt_serves(sms, rows, cols, n) ? ZRoute::kInteger : ZRoute::kLibrary;
}

ZRoute zupdate_route(int sms, int n, int k, int cols, bool integer) {
  if (zblock_small(n, std::max(k, cols))) return ZRoute::kBlock;
  return integer && zcrt_serves(sms, n, cols, k) ? ZRoute::kInteger : ZRoute::kLibrary;
}

void zgram(Runtime& rt, int n, const ZBlock& a, const ZBlock* b, double2* const* c, int count, int ldc, bool upper,
           ZRoute route) {
  GramArgs g{};
  g.a = a;
  g.n = n;
  g.ldc = ldc;
  g.rows = a.cols();
  g.cols = b[0].cols();
  g.upper = upper;
  if (g.rows <= 0 || g.cols <= 0) return;
  const double2 one = make_double2(1, 0), zero = make_double2(0, 0);
  if (route == ZRoute::kInteger && !crt_reserve(rt, crt_plane_bytes(g.rows, n, false), crt_plane_bytes(g.cols, n, true),
                                                crt_result_bytes(rt.sms, g.rows, g.cols, n)))
    route = ZRoute::kLibrary;
  if (route == ZRoute::kLibrary) {
    for (int i = 0; i < count; ++i) {
      double2* const right = c[i] + (long long)b[i].c1 * ldc;   // columns of the second buffer
      gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, a.c1, b[i].c1, n, one, a.p1, n, b[i].p1, n, zero, c[i], ldc);
      gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, a.c1, b[i].c2, n, one, a.p1, n, b[i].p2, n, zero, right, ldc);
      if (!upper) gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, a.c2, b[i].c1, n, one, a.p2, n, b[i].p1, n, zero, c[i] + a.c1, ldc);
      gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, a.c2, b[i].c2, n, one, a.p2, n, b[i].p2, n, zero, right + a.c1, ldc);
    }
    return;
  }
  if (route == ZRoute::kInteger) {
    const CrtPlanes pa = crt_prepare(rt, side_of(a, n, true, true), false, rt.crt_a);   // shared by the products
    for (int i = 0; i < count; ++i) {
      const CrtPlanes pb = crt_prepare(rt, side_of(b[i], n, true, false), true, rt.crt_b);
      crt_product(rt, pa, pb, one, zero, c[i], ldc, upper);
    }
    return;
  }
  for (int i = 0; i < count; ++i) {
    g.b[i] = b[i];
    g.c[i] = c[i];
  }
  g.tiles_i = ceil_div(g.rows, kT);
  g.tiles_j = ceil_div(g.cols, kT);
  g.tiles = upper ? g.tiles_j * (g.tiles_j + 1) / 2 : g.tiles_i * g.tiles_j;
  const int tiles = g.tiles * count;
  // about four CTAs per SM, down to slices of one chunk
  const int chunks = ceil_div(n, kGramK);
  int slices = std::max(1, std::min({ceil_div(4 * rt.sms, tiles), chunks, 64}));
  const int kper = ceil_div(chunks, slices) * kGramK;
  slices = ceil_div(n, kper);
  const size_t need = slices > 1 ? size_t(slices) * tiles * kT * kT : 0;
  if (rt.zwork.size() < need) rt.zwork.resize(need);
  raise_smem_limit(zgram_kernel, kGramSmem);
  launch_chained(dim3(tiles, slices), kGramThreads, kGramSmem, rt.stream, zgram_kernel,
      g, kper, slices, rt.zwork.get());
  HALF_LAUNCH("block Gram products");
  ++rt.prof.launches;
  if (slices > 1) {
    launch_chained(4 * tiles, 256, 0, rt.stream, zgram_reduce_kernel,
        g, slices, rt.zwork.get());
    HALF_LAUNCH("block Gram reduction");
    ++rt.prof.launches;
  }
}

void zupdate(Runtime& rt, int n, const ZBlock* z, const double2* y, int ldy, double2* const* c, int cols, int count,
             double alpha, double beta, ZRoute route) {
  if (n <= 0 || cols <= 0) return;
  const int k = z[0].cols();
  if (route == ZRoute::kInteger && !crt_reserve(rt, crt_plane_bytes(n, k, false), crt_plane_bytes(cols, k, true),
                                                crt_result_bytes(rt.sms, n, cols, k)))
    route = ZRoute::kLibrary;
  if (route == ZRoute::kLibrary) {
    const double2 al = make_double2(alpha, 0), one = make_double2(1, 0);
    for (int i = 0; i < count; ++i) {
      const ZBlock& b = z[i];
      gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, cols, b.c1, al, b.p1, n, y, ldy, make_double2(beta, 0), c[i], n);
      if (b.c2 > 0) gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, n, cols, b.c2, al, b.p2, n, y + b.c1, ldy, one, c[i], n);
    }
    return;
  }
  if (route == ZRoute::kInteger) {
    CrtSide ys;
    ys.p = y;
    ys.ld = ldy;
    ys.rows = cols;
    ys.k = z[0].cols();
    ys.kcontig = true;
    const CrtPlanes py = crt_prepare(rt, ys, true, rt.crt_b);   // shared by the blocks
    for (int i = 0; i < count; ++i) {
      const CrtPlanes pz = crt_prepare(rt, side_of(z[i], n, false, false), false, rt.crt_a);
      crt_product(rt, pz, py, make_double2(alpha, 0), make_double2(beta, 0), c[i], n);
    }
    return;
  }
  UpdateArgs u{};
  for (int i = 0; i < count; ++i) {
    u.z[i] = z[i];
    u.c[i] = c[i];
  }
  u.y = y;
  u.n = n;
  u.ldy = ldy;
  u.cols = cols;
  u.alpha = alpha;
  u.beta = beta;
  raise_smem_limit(zupdate_kernel, kUpSmem);
  launch_chained(dim3(ceil_div(n, kUpRows), ceil_div(cols, kT), count), kUpThreads, kUpSmem, rt.stream, zupdate_kernel,
      u);
  HALF_LAUNCH("block update");
  ++rt.prof.launches;
}

}  // namespace hb
