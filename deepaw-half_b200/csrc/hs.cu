// The matrix-free MIMIC_US H/S operator of one k point.
//
// Reference: apply_hs_operator_cuda (src/half_cuda_assembly.cuf:468-519)
// scatters each band into a zeroed N_r box, runs one cuFFT per band inverse,
// multiplies by Veff/N_r, one cuFFT per band forward, gathers and adds T psi,
// then per species runs three ZGEMMs around a D/Q mixing kernel.
//
// B200 design: the local part is three fused kernels over x-planes of the box
// that never materialise empty data.  Planes are indexed by g1 in the
// sphere's x-extent only (about 40% of the box); within a plane only the rows
// that hold sphere points are transformed along z.
//   K1  sphere -> planes: scatter band points straight into the transform's
//       digit-reversed slots, inverse z FFT on occupied rows, inverse y FFT
//       on all columns, one coalesced plane store;
//   K2  x lines: gather the occupied x slots, inverse x FFT, multiply by
//       Veff/N_r, forward x FFT, store the occupied slots back;
//   K3  planes -> sphere: forward y FFT, forward z FFT on occupied rows,
//       gather sphere points, H psi = . + T psi, S psi = psi.
// Bands go through in chunks (the ACC block size) so the plane buffer of a
// chunk stays resident in the 126 MB L2 between the three kernels.  The
// projector part is one GEMM B^H X over all species and bands, a D/Q mixing
// kernel and the GEMMs accumulating B DY into H X and B QY into S X.  In FP64
// B is stored and the GEMMs are cuBLAS ZGEMM (the reference's calls) or, large
// ones of a mixed solve's FP64 phase, integer products (zcrt.cu); in FP32
// one pass per k point generates B from a radial-angular table
// (Omega^-1/2 beta_l(|q|) Y_lm, one row per species channel), the packed
// plane-wave indices and the ions' b_j.R / 2 pi straight into the bf16 planes
// of the tensor-core GEMM (tc_gemm.cu), in both orientations (conj(B)^T and
// B; 8 bytes per element each), and B [DY | QY] is one GEMM with a doubled N
// writing H X and S X.
#include <algorithm>
#include <cmath>
#include <map>

#include "blas.h"
#include "context.h"
#include "tune.h"
#include "zcrt.h"

namespace hb {

template <typename R>
struct KOperator {
  using C = cplx_t<R>;
  int npw = 0, n1 = 0, n2 = 0, n3 = 0, g1min = 0, nplanes = 0, np = 0, max_rows = 0;
  AxisPlan ax, ay, az;
  DeviceBuffer<int> plane_start, spos, row_start, row_list, slot_plane;
  DeviceBuffer<C> tw;        // exp(-2 pi i t / n) of the x, y and z axes, one after another
  DeviceBuffer<R> veff;      // Veff / N_r, C order
  DeviceBuffer<R> kinetic;
  DeviceBuffer<C> work;      // chunk x nplanes x n2 x n3
  int work_chunk = 0;
  DeviceBuffer<C> B;         // FP64: npw x np, column-major
  // FP64 operator of a mixed solve: its projector products may run on the
  // integer tensor cores (zcrt.cu).  B^H and B in residue planes, made by the
  // first application large enough to use them
  bool integer = false;
  DeviceBuffer<unsigned char> crt_bh_store, crt_b_store;
  CrtPlanes crt_bh, crt_b;
  // FP32: the projector matrix is generated from these tables straight into
  // the bf16 planes of the tensor-core GEMM (tc_gemm.cu), once per k point,
  // in the two orientations the products use
  DeviceBuffer<float> ftab;  // [frow][npw] Omega^-1/2 beta_l(|q|) Y_lm(q^), frow = (species, channel, m)
  DeviceBuffer<unsigned char> bh_store, b_store;
  TcOperand bh_planes;       // conj(B)^T: np x npw
  TcOperand b_planes;        // B: npw x np
  DeviceBuffer<R> dall, qall;            // D per atom, Q per species
  DeviceBuffer<int> col_base, col_a, col_nlm, col_dofs, col_qofs;
  DeviceBuffer<C> coeff, dy, qy;
  int ws_cols = 0;
};

KOperatorSet::~KOperatorSet() = default;

namespace {

constexpr int kXTile = 16;
constexpr int kPlaneThreads = 512;

template <typename C>
__device__ __forceinline__ C czero() { C c; c.x = 0; c.y = 0; return c; }

// The local operator's three kernels are bound by instruction issue (half of
// the slots in FP32) and the latency between passes, not by HBM (a chunk's
// planes stay in L2), so every pass over a plane or line that can be saved is:
// the first and last
// transform passes read and write global memory directly, rows known to be
// zero are neither cleared nor loaded, and rows nobody reads are not stored.
// Rows of a plane are padded by one element in shared memory so that the z
// passes, whose threads run over rows, are free of bank conflicts.  Kernel
// time of one mixed solve of the 216-atom cell (96^3 box, B200), against
// four radix <= 5 passes per axis with separate clear, scatter, product and
// gather passes: K2 FP32 96.5 -> 26.7 ms, K2 FP64 67.0 -> 27.1 ms, K1 + K3
// FP32 56.8 -> 27.3 ms, FP64 64.4 -> 28.2 ms.

// Shared memory of a plane kernel: twiddles of both axes, the plane with
// padded rows, the occupied rows and a flag per row.
template <typename R>
size_t plane_smem(int n2, int n3) {
  return (n2 + n3 + size_t(n2) * (n3 + 1)) * sizeof(cplx_t<R>) + size_t(n2) * 2 * sizeof(int);
}

// Threads of a plane kernel: 512 where shared memory holds one plane (FP64)
// or two (FP32) per SM, which is also what the registers allow; smaller
// planes run as more and smaller CTAs of the same total, so that one CTA's
// barriers and loads overlap another's transforms.
template <typename R>
int plane_threads(size_t smem) {
  const int total = sizeof(R) == 4 ? 1024 : 512;   // resident threads per SM (64 / 128 registers)
  int th = kPlaneThreads;
  while (th > 128 && size_t(total / (th / 2)) * (smem + 1024) <= 227 * 1024) th /= 2;
  return th;
}

// Threads of an x-line kernel: one per item of the pass with most items.
inline int xline_threads(const FFTPlan& p) {
  int items = 0;
  for (int s = 0; s < p.nstages; ++s) items = std::max(items, p.n / p.radix[s] * kXTile);
  return std::min(256, (items + 31) / 32 * 32);
}

template <typename R>
struct PlaneSmem {
  using C = cplx_t<R>;
  C *twy, *twz, *plane;
  int *rows, *occ;
  __device__ __forceinline__ PlaneSmem(unsigned char* raw, int n2, int n3) {
    twy = reinterpret_cast<C*>(raw);
    twz = twy + n2;
    plane = twz + n3;
    rows = reinterpret_cast<int*>(plane + size_t(n2) * (n3 + 1));
    occ = rows + n2;
  }
};

// tw: the twiddles of the x, y and z axes one after another.
template <typename R>
__global__ void __launch_bounds__(kPlaneThreads, sizeof(R) == 4 ? 2 : 1)
    k1_sphere_to_planes(const cplx_t<R>* __restrict__ psi, long long ld, int b0, int n2, int n3, int nplanes,
                        const int* __restrict__ plane_start, const int* __restrict__ spos,
                        const int* __restrict__ row_start, const int* __restrict__ row_list, FFTPlan py, FFTPlan pz,
                        const cplx_t<R>* __restrict__ tw_yz, cplx_t<R>* __restrict__ work) {
  wait_previous();
  using C = cplx_t<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneSmem<R> sm(smem_raw, n2, n3);
  C* const plane = sm.plane;
  const int n3p = n3 + 1;
  const int j = blockIdx.x, b = blockIdx.y;
  for (int t = threadIdx.x; t < n2 + n3; t += blockDim.x) sm.twy[t] = tw_yz[t];
  const int r0 = row_start[j], nrows = row_start[j + 1] - r0;
  for (int t = threadIdx.x; t < n2; t += blockDim.x) sm.occ[t] = 0;
  for (int r = threadIdx.x >> 5; r < nrows; r += blockDim.x >> 5) {   // one warp per occupied row
    const int row = row_list[r0 + r];
    if ((threadIdx.x & 31) == 0) sm.rows[r] = row * n3p;
    for (int t = threadIdx.x & 31; t < n3; t += 32) plane[row * n3p + t] = czero<C>();
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nrows; t += blockDim.x) sm.occ[sm.rows[t] / n3p] = 1;
  const C* col = psi + (long long)(b0 + b) * ld;
  const int p0 = plane_start[j], p1 = plane_start[j + 1];
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) plane[spos[p]] = col[p];
  __syncthreads();
  const int* const rows = sm.rows;
  for (int s = pz.nstages - 1; s >= 0; --s) {
    fft_pass<true, +1, C, R>(
        pz, s, nrows, sm.twz, [&](int p, int i) { return plane[rows[p] + i]; },
        [&](int p, int i, C v) { plane[rows[p] + i] = v; });
    __syncthreads();
  }
  C* const dst = work + ((long long)b * nplanes + j) * n2 * n3;
  const int* const occ = sm.occ;
  auto ld_occ = [&](int p, int i) { return occ[i] ? plane[i * n3p + p] : czero<C>(); };
  auto st_plane = [&](int p, int i, C v) { plane[i * n3p + p] = v; };
  auto st_work = [&](int p, int i, C v) { dst[i * n3 + p] = v; };
  if (py.nstages == 1) {
    fft_pass<true, +1, C, R>(py, 0, n3, sm.twy, ld_occ, st_work);
    return;
  }
  fft_pass<true, +1, C, R>(py, py.nstages - 1, n3, sm.twy, ld_occ, st_plane);
  __syncthreads();
  auto ld_plane = [&](int p, int i) { return plane[i * n3p + p]; };
  if (py.nstages == 3) {
    fft_pass<true, +1, C, R>(py, 1, n3, sm.twy, ld_plane, st_plane);
    __syncthreads();
  }
  fft_pass<true, +1, C, R>(py, 0, n3, sm.twy, ld_plane, st_work);
}

// Shared memory of an x-line kernel: twiddles, the tile's box points, one
// real per point (Veff / N_r, or the density) and the plane of each slot.
template <typename R>
size_t xline_smem(int n1) {
  return (n1 + size_t(n1) * kXTile) * sizeof(cplx_t<R>) + size_t(n1) * kXTile * sizeof(R) + size_t(n1) * sizeof(int);
}

// One CTA per (i2, z tile) and group of bands_per_cta of the chunk's nb
// bands, looping over its bands: the twiddles, the plane of every slot
// (slot_plane, -1 where the sphere has none) and the tile's Veff are set up
// once per CTA.  Per band, three passes for a two-pass axis: the first
// inverse pass loads the occupied planes from global memory, the last
// inverse pass, the product with Veff and the first forward pass are one
// pass in registers, and the last forward pass stores the occupied planes.
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 2) k2_xlines(cplx_t<R>* __restrict__ work, int n1, int n2, int n3, int nplanes,
                                                 const int* __restrict__ slot_plane, FFTPlan px,
                                                 const cplx_t<R>* __restrict__ tw_x, const R* __restrict__ veff, int nb,
                                                 int bands_per_cta) {
  wait_previous();
  using C = cplx_t<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const tw = reinterpret_cast<C*>(smem_raw);
  C* const X = tw + n1;                                      // [slot][tz]
  R* const vt = reinterpret_cast<R*>(X + n1 * kXTile);       // [i1][tz] Veff / N_r
  int* const slot = reinterpret_cast<int*>(vt + n1 * kXTile);
  const int tiles = (n3 + kXTile - 1) / kXTile;
  const int i2 = blockIdx.x / tiles, z0 = (blockIdx.x - i2 * tiles) * kXTile;
  const int nz = min(kXTile, n3 - z0);
  const int npl = n2 * n3;
  for (int t = threadIdx.x; t < n1; t += blockDim.x) {
    tw[t] = tw_x[t];
    const int jj = slot_plane[t];
    slot[t] = jj < 0 ? -1 : jj * npl;
  }
  for (int t = threadIdx.x; t < n1 * kXTile; t += blockDim.x) {
    const int i1 = t / kXTile, c = t - i1 * kXTile;
    vt[t] = c < nz ? veff[((long long)i1 * n2 + i2) * n3 + z0 + c] : R(0);
  }
  __syncthreads();
  auto ld_x = [&](int p, int i) { return X[i * kXTile + p]; };
  auto st_x = [&](int p, int i, C v) { X[i * kXTile + p] = v; };
  auto times_v = [&](int p, int i, C v) { return cscale(v, vt[i * kXTile + p]); };
  const int last = px.nstages - 1;
  const int bend = min(nb, (blockIdx.y + 1) * bands_per_cta);
  for (int b = blockIdx.y * bands_per_cta; b < bend; ++b) {
    C* const base = work + (long long)b * nplanes * npl + (long long)i2 * n3 + z0;
    auto ld_work = [&](int p, int i) {
      const int o = slot[i];
      return o >= 0 && p < nz ? base[o + p] : czero<C>();
    };
    auto st_work = [&](int p, int i, C v) {
      const int o = slot[i];
      if (o >= 0 && p < nz) base[o + p] = v;
    };
    if (last == 0) {
      fft_pass_fused<C, R>(px, kXTile, tw, ld_work, times_v, st_work);
      continue;
    }
    fft_pass<true, +1, C, R>(px, last, kXTile, tw, ld_work, st_x);
    __syncthreads();
    if (last == 2) {
      fft_pass<true, +1, C, R>(px, 1, kXTile, tw, ld_x, st_x);
      __syncthreads();
    }
    fft_pass_fused<C, R>(px, kXTile, tw, ld_x, times_v, st_x);
    __syncthreads();
    if (last == 2) {
      fft_pass<false, -1, C, R>(px, 1, kXTile, tw, ld_x, st_x);
      __syncthreads();
    }
    fft_pass<false, -1, C, R>(px, last, kXTile, tw, ld_x, st_work);
    __syncthreads();
  }
}

template <typename R>
__global__ void __launch_bounds__(kPlaneThreads, sizeof(R) == 4 ? 2 : 1)
    k3_planes_to_sphere(const cplx_t<R>* __restrict__ work, int n2, int n3, int nplanes,
                        const int* __restrict__ plane_start, const int* __restrict__ spos,
                        const int* __restrict__ row_start, const int* __restrict__ row_list, FFTPlan py, FFTPlan pz,
                        const cplx_t<R>* __restrict__ tw_yz, const cplx_t<R>* __restrict__ psi, long long ld, int b0,
                        const R* __restrict__ kinetic, cplx_t<R>* __restrict__ hpsi, cplx_t<R>* __restrict__ spsi) {
  wait_previous();
  using C = cplx_t<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneSmem<R> sm(smem_raw, n2, n3);
  C* const plane = sm.plane;
  const int n3p = n3 + 1;
  const int j = blockIdx.x, b = blockIdx.y;
  for (int t = threadIdx.x; t < n2 + n3; t += blockDim.x) sm.twy[t] = tw_yz[t];
  const int r0 = row_start[j], nrows = row_start[j + 1] - r0;
  for (int t = threadIdx.x; t < n2; t += blockDim.x) sm.occ[t] = 0;
  __syncthreads();
  for (int t = threadIdx.x; t < nrows; t += blockDim.x) {
    const int row = row_list[r0 + t];
    sm.rows[t] = row * n3p;
    sm.occ[row] = 1;
  }
  const C* const src = work + ((long long)b * nplanes + j) * n2 * n3;
  const int* const occ = sm.occ;
  auto ld_work = [&](int p, int i) { return src[i * n3 + p]; };
  auto ld_plane = [&](int p, int i) { return plane[i * n3p + p]; };
  auto st_plane = [&](int p, int i, C v) { plane[i * n3p + p] = v; };
  auto st_occ = [&](int p, int i, C v) { if (occ[i]) plane[i * n3p + p] = v; };
  if (py.nstages == 1) {
    __syncthreads();   // occ
    fft_pass<false, -1, C, R>(py, 0, n3, sm.twy, ld_work, st_occ);
  } else {
    fft_pass<false, -1, C, R>(py, 0, n3, sm.twy, ld_work, st_plane);
    __syncthreads();
    if (py.nstages == 3) {
      fft_pass<false, -1, C, R>(py, 1, n3, sm.twy, ld_plane, st_plane);
      __syncthreads();
    }
    fft_pass<false, -1, C, R>(py, py.nstages - 1, n3, sm.twy, ld_plane, st_occ);
  }
  __syncthreads();
  const int* const rows = sm.rows;
  for (int s = 0; s < pz.nstages; ++s) {
    fft_pass<false, -1, C, R>(
        pz, s, nrows, sm.twz, [&](int p, int i) { return plane[rows[p] + i]; },
        [&](int p, int i, C v) { plane[rows[p] + i] = v; });
    __syncthreads();
  }
  const long long off = (long long)(b0 + b) * ld;
  const int p0 = plane_start[j], p1 = plane_start[j + 1];
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    C x = psi[off + p];
    C h = plane[spos[p]];
    R kin = kinetic[p];
    h.x += kin * x.x;
    h.y += kin * x.y;
    hpsi[off + p] = h;
    spsi[off + p] = x;
  }
}

// Density variant of k2_xlines: the block owns the box points (all i1, its
// i2, its z tile) and runs the chunk's bands in order through the inverse x
// transform, accumulating bw[b] |psi_b(r)|^2; the chunk total is added to
// density (C order) once.  No atomics: each point has one owner.
__global__ void __launch_bounds__(256) k2_density(const double2* __restrict__ work, int n1, int n2, int n3,
                                                  int nplanes, const int* __restrict__ slot_plane, FFTPlan px,
                                                  const double2* __restrict__ tw_x, const double* __restrict__ bw,
                                                  int nb, double* __restrict__ density) {
  using C = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const tw = reinterpret_cast<C*>(smem_raw);
  C* const X = tw + n1;                                              // [slot][tz]
  double* const acc = reinterpret_cast<double*>(X + n1 * kXTile);    // [i1][tz]
  int* const slot = reinterpret_cast<int*>(acc + n1 * kXTile);
  const int tiles = (n3 + kXTile - 1) / kXTile;
  const int i2 = blockIdx.x / tiles, z0 = (blockIdx.x - i2 * tiles) * kXTile;
  const int nz = min(kXTile, n3 - z0);
  const int npl = n2 * n3;
  for (int t = threadIdx.x; t < n1; t += blockDim.x) {
    tw[t] = tw_x[t];
    const int jj = slot_plane[t];
    slot[t] = jj < 0 ? -1 : jj * npl;
  }
  for (int t = threadIdx.x; t < n1 * kXTile; t += blockDim.x) acc[t] = 0.0;
  __syncthreads();
  auto ld_x = [&](int p, int i) { return X[i * kXTile + p]; };
  auto st_x = [&](int p, int i, C v) { X[i * kXTile + p] = v; };
  const int last = px.nstages - 1;
  for (int b = 0; b < nb; ++b) {
    const C* const base = work + (long long)b * nplanes * npl + (long long)i2 * n3 + z0;
    const double w = bw[b];
    auto ld_work = [&](int p, int i) {
      const int o = slot[i];
      return o >= 0 && p < nz ? base[o + p] : czero<C>();
    };
    // every pass maps points to threads alike, so each sum has one writer
    auto add = [&](int p, int i, C v) { acc[i * kXTile + p] += w * (v.x * v.x + v.y * v.y); };
    if (last == 0) {
      fft_pass<true, +1, C, double>(px, 0, kXTile, tw, ld_work, add);
      continue;
    }
    fft_pass<true, +1, C, double>(px, last, kXTile, tw, ld_work, st_x);
    __syncthreads();
    if (last == 2) {
      fft_pass<true, +1, C, double>(px, 1, kXTile, tw, ld_x, st_x);
      __syncthreads();
    }
    fft_pass<true, +1, C, double>(px, 0, kXTile, tw, ld_x, add);
    __syncthreads();
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n1 * kXTile; t += blockDim.x) {
    int i1 = t / kXTile, c = t - i1 * kXTile;
    if (c < nz) density[((long long)i1 * n2 + i2) * n3 + z0 + c] += acc[t];
  }
}

// dy[:,b] = blockdiag(D_atom) coeff[:,b], qy[:,b] = blockdiag(Q_species) coeff[:,b]
// (src/half_cuda_assembly.cuf:220-237)
template <typename R>
__global__ void mix_kernel(const cplx_t<R>* __restrict__ coeff, int np, int nb, const int* __restrict__ col_base,
                           const int* __restrict__ col_a, const int* __restrict__ col_nlm,
                           const int* __restrict__ col_dofs, const int* __restrict__ col_qofs,
                           const R* __restrict__ dall, const R* __restrict__ qall, cplx_t<R>* __restrict__ dy,
                           cplx_t<R>* __restrict__ qy) {
  after_previous();
  using C = cplx_t<R>;
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)np * nb) return;
  int p = int(idx % np);
  long long b = idx / np;
  const int base = col_base[p], a = col_a[p], nlm = col_nlm[p];
  const R* drow = dall + col_dofs[p] + a * nlm;
  const R* qrow = qall + col_qofs[p] + a * nlm;
  const C* c = coeff + b * np + base;
  C zd = czero<C>(), zq = czero<C>();
  for (int k = 0; k < nlm; ++k) {
    C v = c[k];
    zd.x += drow[k] * v.x; zd.y += drow[k] * v.y;
    zq.x += qrow[k] * v.x; zq.y += qrow[k] * v.y;
  }
  dy[idx] = zd;
  qy[idx] = zq;
}

struct ProjCol {
  int chan;      // global channel index into the radial tables
  int l, m;
  int ion;
  double gmax;
};

// beta_l(|q|) Y_lm(q^) of one projector channel at one plane wave, with the
// reference's 0.99 gmax cut (src/half_paw.F90:52-65).
__device__ __forceinline__ double radial_angular(const ProjCol& col, double qx, double qy, double qz,
                                                 const double* __restrict__ ry, const double* __restrict__ rm2) {
  double qn = sqrt(qx * qx + qy * qy + qz * qz);
  double theta = 0, phi = 0;
  if (qn > 1.0e-10) {
    theta = acos(fmax(-1.0, fmin(1.0, qz / qn)));
    phi = atan2(qy, qx);
  }
  double rval = spline_eval(ry + col.chan * 100, rm2 + col.chan * 100, 100, col.gmax, qn);
  if (qn > 0.99 * col.gmax) rval = 0;
  return rval * real_ylm(col.l, col.m, cos(theta), phi);
}

// B[g, p] = Omega^-1/2 (-i)^l beta_l(|q|) Y_lm(q^) exp(-i q.R)   (src/half_paw.F90:52-65)
// One thread per (plane wave, atom): the phase once, the radial-angular
// factors from the table that the atoms of a species share.  Evaluating
// spline, harmonics and phase per element took 151 us for the 64-atom cell
// (512 projectors, 11,000 plane waves, 90 MB written), this kernel 18 us and
// the table 5 us.
__global__ void projector_kernel(double2* __restrict__ B, int npw, const double* __restrict__ q,
                                 const double* __restrict__ ftab, const int* __restrict__ pcol,
                                 const int2* __restrict__ atom_cols, const double* __restrict__ pos) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x, ion = blockIdx.y;
  if (g >= npw) return;
  const int2 cols = atom_cols[ion];   // first column, columns
  const double ph = q[3 * g] * pos[3 * ion] + q[3 * g + 1] * pos[3 * ion + 1] + q[3 * g + 2] * pos[3 * ion + 2];
  double s, c;
  sincos(ph, &s, &c);
  for (int p = cols.x; p < cols.x + cols.y; ++p) {
    const int d = pcol[p];
    const double amp = ftab[(long long)((d >> 2) & 0x3FFF) * npw + g];
    // (-i)^l * (cos - i sin)
    const double re = amp * c, im = -amp * s;
    double tr, ti;
    switch (d & 3) {
      case 0: tr = re; ti = im; break;
      case 1: tr = im; ti = -re; break;
      case 2: tr = -re; ti = -im; break;
      default: tr = -im; ti = re; break;
    }
    B[(long long)p * npw + g] = make_double2(tr, ti);
  }
}

// ftab[r][g] = Omega^-1/2 beta_l(|q|) Y_lm(q^) for the channel rows of the
// generated FP32 projector tiles (one row per (species, channel, m)).
__global__ void radial_angular_table_kernel(double* __restrict__ ftab, int npw, const double* __restrict__ q,
                                            const ProjCol* __restrict__ rows, const double* __restrict__ ry,
                                            const double* __restrict__ rm2, double pref) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  int r = blockIdx.y;
  if (g >= npw) return;
  ftab[(long long)r * npw + g] = pref * radial_angular(rows[r], q[3 * g], q[3 * g + 1], q[3 * g + 2], ry, rm2);
}

template <typename R>
__global__ void scale_copy_kernel(const double* __restrict__ in, R* __restrict__ out, long long n, double s) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = R(in[i] * s);
}

struct HostGeom {
  int g1min = 0, nplanes = 0, max_rows = 0;
  std::vector<int> plane_start, spos, row_start, row_list;
  std::vector<int> slot_plane;   // plane of each x slot, -1 where the sphere has none
};

HostGeom plane_geometry(const Basis& b, const AxisPlan& ax, const AxisPlan& ay, const AxisPlan& az) {
  HostGeom h;
  const int n1 = b.shape[0], n2 = b.shape[1], n3 = b.shape[2];
  const long long npw = b.npw();
  int g1min = b.gvec[0], g1max = b.gvec[3 * (npw - 1)];
  h.g1min = g1min;
  h.nplanes = g1max - g1min + 1;
  if (h.nplanes > n1) fail(kInternal, "sphere x-extent exceeds the FFT box");
  h.plane_start.assign(h.nplanes + 1, 0);
  h.slot_plane.assign(n1, -1);
  h.spos.resize(npw);
  long long p = 0;
  for (int j = 0; j < h.nplanes; ++j) {
    h.plane_start[j] = int(p);
    h.row_start.push_back(int(h.row_list.size()));
    int last_i2 = -1;
    while (p < npw && b.gvec[3 * p] == g1min + j) {
      int i2 = ((b.gvec[3 * p + 1] % n2) + n2) % n2, i3 = ((b.gvec[3 * p + 2] % n3) + n3) % n3;
      int row = ay.pos[i2];
      if (i2 != last_i2) { h.row_list.push_back(row); last_i2 = i2; }
      h.spos[p] = row * (n3 + 1) + az.pos[i3];   // rows are padded in shared memory
      ++p;
    }
    int i1 = (((g1min + j) % n1) + n1) % n1;
    h.slot_plane[ax.pos[i1]] = j;
  }
  h.plane_start[h.nplanes] = int(p);
  h.row_start.push_back(int(h.row_list.size()));
  // z passes: threads run over a plane's rows, so neighbours in the list get
  // different shared-memory banks where the occupied rows allow it
  std::vector<int> by_bank;
  for (int j = 0; j < h.nplanes; ++j) {
    const int a = h.row_start[j], e = h.row_start[j + 1];
    by_bank.assign(h.row_list.begin() + a, h.row_list.begin() + e);
    std::sort(by_bank.begin(), by_bank.end(), [](int x, int y) { return x % 16 != y % 16 ? x % 16 < y % 16 : x < y; });
    // deal the banks' rows out in turn: the i-th row of every bank, then the next
    int start[17] = {};
    for (int r : by_bank) ++start[r % 16 + 1];
    for (int i = 0; i < 16; ++i) start[i + 1] += start[i];
    for (int i = 0, o = a; o < e; ++i)
      for (int bk = 0; bk < 16; ++bk)
        if (start[bk] + i < start[bk + 1]) h.row_list[o++] = by_bank[start[bk] + i];
    h.max_rows = std::max(h.max_rows, e - a);
  }
  if (p != npw) fail(kInternal, "basis is not ordered by g1");
  return h;
}

// What generates projector elements: one radial-angular row per (species,
// channel, m), the column descriptors, the packed plane-wave indices and the
// ions' b_j.R / 2 pi.
struct ProjGen {
  std::vector<ProjCol> frows;
  std::vector<int> pcol, gpack;
  std::vector<double> afrac;
};

// The projector columns' tables: first column of a column's atom, its place
// in the atom, the atom's column count, offsets of D and Q.
struct ProjTables {
  std::vector<int> base, a, nlm, dofs, qofs;
};

// Sizes and small tables of one precision's operator; the tables are on the
// device once the batch is flushed.
template <typename R>
void stage_operator(Context& ctx, const Basis& basis, const HostGeom& hg, int np, const ProjTables& pt,
                    UploadBatch& batch, KOperator<R>& op) {
  using C = cplx_t<R>;
  op.npw = int(basis.npw());
  op.n1 = basis.shape[0]; op.n2 = basis.shape[1]; op.n3 = basis.shape[2];
  op.ax = make_axis_plan(op.n1); op.ay = make_axis_plan(op.n2); op.az = make_axis_plan(op.n3);
  op.g1min = hg.g1min; op.nplanes = hg.nplanes; op.max_rows = hg.max_rows; op.np = np;
  if (plane_smem<R>(op.n2, op.n3) > 227 * 1024)
    fail(kUnavailable, "FFT plane " + std::to_string(op.n2) + "x" + std::to_string(op.n3) +
                           " exceeds the shared-memory capacity of one CTA at this precision");
  batch.add(op.plane_start, hg.plane_start);
  batch.add(op.spos, hg.spos);
  batch.add(op.row_start, hg.row_start);
  batch.add(op.row_list, hg.row_list);
  batch.add(op.slot_plane, hg.slot_plane);
  std::vector<C> tw;
  const int axes[3] = {op.n1, op.n2, op.n3};
  for (int a = 0; a < 3; ++a)
    for (int t = 0; t < axes[a]; ++t)
      tw.push_back(cmake(R(std::cos(2.0 * kPi * t / axes[a])), R(-std::sin(2.0 * kPi * t / axes[a]))));
  batch.add(op.tw, tw);
  batch.add(op.kinetic, std::vector<R>(basis.kinetic.begin(), basis.kinetic.end()));
  std::vector<R> dall, qall;
  for (auto& sp : ctx.species) {
    dall.insert(dall.end(), sp.dij_host.begin(), sp.dij_host.end());
    qall.insert(qall.end(), sp.qij_host.begin(), sp.qij_host.end());
  }
  batch.add(op.dall, dall);
  batch.add(op.qall, qall);
  batch.add(op.col_base, pt.base);
  batch.add(op.col_a, pt.a);
  batch.add(op.col_nlm, pt.nlm);
  batch.add(op.col_dofs, pt.dofs);
  batch.add(op.col_qofs, pt.qofs);
}

// The operator's large tables, on the device.
template <typename R>
void fill_operator(Context& ctx, Runtime& rt, KOperatorSet& ks, int nfrows, DeviceBuffer<double2>& B64,
                   KOperator<R>& op) {
  cudaStream_t s = rt.stream;
  const long long nr = ctx.nr();
  op.veff.resize(nr);
  scale_copy_kernel<R><<<ceil_div(nr, 256), 256, 0, s>>>(ctx.veff.get(), op.veff.get(), nr, 1.0 / double(nr));
  if constexpr (sizeof(R) == 8) {
    op.B = std::move(B64);   // only the FP64 operator reads the stored matrix
  } else if (op.np > 0) {
    const long long nt = (long long)nfrows * op.npw;
    op.ftab.resize(size_t(nt));
    scale_copy_kernel<float><<<ceil_div(nt, 256), 256, 0, s>>>(ks.ftab64.get(), op.ftab.get(), nt, 1.0);
    HALF_LAUNCH("radial-angular table (FP32)");
    TcOperand g;
    g.kind = TcOperand::kProjConj;
    g.rows = op.np;
    g.kdim = op.npw;
    g.ftab = op.ftab.get();
    g.gpack = ks.gpack.get();
    g.pcol = ks.pcol.get();
    g.afrac = ks.afrac.get();
    g.kf0 = ks.kf[0];
    g.kf1 = ks.kf[1];
    g.kf2 = ks.kf[2];
    g.npw = op.npw;
    op.bh_planes = tc_presplit_a(rt, g, op.bh_store);
    g.kind = TcOperand::kProj;
    g.rows = op.npw;
    g.kdim = op.np;
    op.b_planes = tc_presplit_a(rt, g, op.b_store);
  }
  HALF_LAUNCH("operator tables");
  raise_smem_limit(k1_sphere_to_planes<R>, plane_smem<R>(op.n2, op.n3));
  raise_smem_limit(k3_planes_to_sphere<R>, plane_smem<R>(op.n2, op.n3));
  raise_smem_limit(k2_xlines<R>, xline_smem<R>(op.n1));
}

}  // namespace

std::unique_ptr<KOperatorSet> prepare_operator(Context& ctx, Runtime& rt, const double k[3], bool fp64, bool fp32) {
  auto ks = std::make_unique<KOperatorSet>();
  ks->rt = &rt;
  ks->basis = build_basis(ctx.crystal, ctx.charge.shape, ctx.encut, k);
  const Basis& basis = ks->basis;
  const int npw = int(basis.npw());
  if (npw < 1) fail(kInvalidArgument, "empty plane-wave basis");
  cudaStream_t s = rt.stream;
  AxisPlan ax = make_axis_plan(basis.shape[0]), ay = make_axis_plan(basis.shape[1]), az = make_axis_plan(basis.shape[2]);
  HostGeom hg = plane_geometry(basis, ax, ay, az);
  // projector columns: species-major, atom-major, then (channel, m)
  std::vector<ProjCol> cols;
  ProjTables pt;
  std::vector<int2> atom_cols(ctx.crystal.nions(), make_int2(0, 0));   // first column and columns per ion
  std::vector<double> ry, rm2, pos;
  int chan0 = 0, dofs = 0, qofs = 0, col0 = 0;
  for (auto& sp : ctx.species) {
    for (int a = 0; a < sp.natoms; ++a) {
      int ilm = 0;
      atom_cols[sp.first_ion + a] = make_int2(col0 + a * sp.nlm, sp.nlm);
      for (int c = 0; c < sp.nchan; ++c) {
        int l = sp.lps[c];
        for (int m = -l; m <= l; ++m, ++ilm) {
          cols.push_back({chan0 + c, l, m, sp.first_ion + a, sp.pspnl_gmax});
          pt.base.push_back(col0 + a * sp.nlm);
          pt.a.push_back(ilm);
          pt.nlm.push_back(sp.nlm);
          pt.dofs.push_back(dofs + a * sp.nlm * sp.nlm);
          pt.qofs.push_back(qofs);
        }
      }
    }
    ry.insert(ry.end(), sp.radial_y.begin(), sp.radial_y.end());
    rm2.insert(rm2.end(), sp.radial_m2.begin(), sp.radial_m2.end());
    chan0 += sp.nchan;
    dofs += sp.natoms * sp.nlm * sp.nlm;
    qofs += sp.nlm * sp.nlm;
    col0 += sp.natoms * sp.nlm;
  }
  for (int i = 0; i < ctx.crystal.nions(); ++i) {
    auto r = ctx.crystal.cartesian(i);
    pos.insert(pos.end(), r.begin(), r.end());
  }
  const int np = int(cols.size());
  ks->np = np;
  // generated-tile tables for the FP32 operator: radial-angular rows are per
  // (species, channel, m), shared by the species' atoms
  ProjGen gen;
  {
    int chan = 0, frow0 = 0;
    size_t c = 0;
    for (auto& sp : ctx.species) {
      for (int ch = 0; ch < sp.nchan; ++ch) {
        int l = sp.lps[ch];
        for (int m = -l; m <= l; ++m) gen.frows.push_back({chan + ch, l, m, 0, sp.pspnl_gmax});
      }
      for (int a = 0; a < sp.natoms; ++a)
        for (int ilm = 0; ilm < sp.nlm; ++ilm, ++c) {
          if (cols[c].ion >= (1 << 15) || frow0 + ilm >= (1 << 14)) fail(kUnavailable, "too many ions or projector channels");
          gen.pcol.push_back((cols[c].ion << 16) | ((frow0 + ilm) << 2) | (cols[c].l & 3));
        }
      chan += sp.nchan;
      frow0 += sp.nlm;
    }
    auto rec = ctx.crystal.reciprocal();
    for (int i = 0; i < ctx.crystal.nions(); ++i) {
      auto r = ctx.crystal.cartesian(i);
      for (int j = 0; j < 3; ++j)
        gen.afrac.push_back((rec[3 * j] * r[0] + rec[3 * j + 1] * r[1] + rec[3 * j + 2] * r[2]) / (2.0 * kPi));
    }
  }
  for (size_t g = 0; g < basis.gvec.size(); ++g)
    if (basis.gvec[g] < -512 || basis.gvec[g] > 511) fail(kUnavailable, "plane-wave index beyond the packed range");
  gen.gpack.resize(npw);
  for (int g = 0; g < npw; ++g)
    gen.gpack[g] = (basis.gvec[3 * g] & 1023) | ((basis.gvec[3 * g + 1] & 1023) << 10) |
                   ((basis.gvec[3 * g + 2] & 1023) << 20);
  for (int j = 0; j < 3; ++j) ks->kf[j] = basis.kpoint[j];
  // every small table in one copy
  UploadBatch batch;
  DeviceBuffer<double> dry, drm2, dpos;
  DeviceBuffer<ProjCol> drows;
  DeviceBuffer<int2> datom;
  batch.add(ks->qvec, basis.qvec);
  batch.add(ks->gpack, gen.gpack);
  batch.add(ks->pcol, gen.pcol);
  batch.add(ks->afrac, gen.afrac);
  batch.add(dry, ry);
  batch.add(drm2, rm2);
  batch.add(dpos, pos);
  batch.add(drows, gen.frows);
  batch.add(datom, atom_cols);
  if (fp64) {
    ks->op64 = std::make_unique<KOperator<double>>();
    ks->op64->integer = fp32;   // both precisions: a mixed solve
    stage_operator<double>(ctx, basis, hg, np, pt, batch, *ks->op64);
  }
  if (fp32) {
    ks->op32 = std::make_unique<KOperator<float>>();
    stage_operator<float>(ctx, basis, hg, np, pt, batch, *ks->op32);
  }
  batch.flush(ks->arena, s);
  DeviceBuffer<double2> B64(fp64 ? (size_t)npw * np : 0);
  const int nf = int(gen.frows.size());
  if (np > 0) {   // projector generation tables, shared by the FP32 operator's planes and the force adjoint
    ks->ftab64.resize(size_t(nf) * npw);
    radial_angular_table_kernel<<<dim3(ceil_div(npw, 256), nf), 256, 0, s>>>(
        ks->ftab64.get(), npw, ks->qvec.get(), drows.get(), dry.get(), drm2.get(), 1.0 / std::sqrt(ctx.crystal.volume()));
    HALF_LAUNCH("radial-angular table");
    if (fp64) {
      projector_kernel<<<dim3(ceil_div(npw, 256), ctx.crystal.nions()), 256, 0, s>>>(
          B64.get(), npw, ks->qvec.get(), ks->ftab64.get(), ks->pcol.get(), datom.get(), dpos.get());
      HALF_LAUNCH("projectors");
    }
  }
  if (fp64) fill_operator<double>(ctx, rt, *ks, nf, B64, *ks->op64);
  if (fp32) fill_operator<float>(ctx, rt, *ks, nf, B64, *ks->op32);
  HALF_CUDA(cudaStreamSynchronize(s));
  return ks;
}

template <typename R>
KOperator<R>& pick(KOperatorSet& ks);
template <>
KOperator<double>& pick<double>(KOperatorSet& ks) {
  if (!ks.op64) fail(kInternal, "FP64 operator not prepared");
  return *ks.op64;
}
template <>
KOperator<float>& pick<float>(KOperatorSet& ks) {
  if (!ks.op32) fail(kInternal, "FP32 operator not prepared");
  return *ks.op32;
}

template <typename R>
void apply_nonlocal(Runtime& rt, KOperator<R>& op, const cplx_t<R>* x, long long ld, int nb, cplx_t<R>* hx,
                    cplx_t<R>* sx);

template <typename R>
void apply_hs(Context& ctx, KOperatorSet& ks, const cplx_t<R>* x, long long ld, int nb, cplx_t<R>* hx, cplx_t<R>* sx,
              int chunk) {
  using C = cplx_t<R>;
  KOperator<R>& op = pick<R>(ks);
  Runtime& rt = *ks.rt;
  cudaStream_t s = rt.stream;
  if (nb <= 0) return;
  // chunk <= 0: bands per chunk chosen by the autotuner (tune.h) per box,
  // sphere extent and precision; every choice gives bit-identical results
  int tune_token = 0, tune_index = 0;
  std::string tune_key;
  if (chunk <= 0) {
    static const std::vector<int> cand = {16, 8, 32, 64};
    tune_key = "local " + std::to_string(op.n1) + "x" + std::to_string(op.n2) + "x" +
                            std::to_string(op.n3) + " planes " + std::to_string(op.nplanes) + " fp" +
                            std::to_string(8 * sizeof(R));
    tune_index = Tuner::pick(tune_key, cand);
    chunk = cand[tune_index];
  }
  chunk = std::max(1, std::min(chunk, nb));
  if (op.work_chunk < chunk) {
    op.work.resize((size_t)chunk * op.nplanes * op.n2 * op.n3);
    op.work_chunk = chunk;
  }
  if (!tune_key.empty()) tune_token = Tuner::begin(tune_key, tune_index, s);   // the kernels alone, no allocation
  const size_t psm = plane_smem<R>(op.n2, op.n3), xsm = xline_smem<R>(op.n1);
  const int pth = plane_threads<R>(psm);
  const int tiles = (op.n3 + kXTile - 1) / kXTile;
  const int sms = rt.sms;
  Profile& pf = rt.prof;
  const int ev_sweep = pf.record(s);
  const int ev_local = ev_sweep;
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    int nbc = std::min(chunk, nb - b0);
    launch_chained(dim3(op.nplanes, nbc), pth, psm, s, k1_sphere_to_planes<R>,
        x, ld, b0, op.n2, op.n3, op.nplanes, op.plane_start.get(), op.spos.get(), op.row_start.get(),
        op.row_list.get(), op.ay.plan, op.az.plan, op.tw.get() + op.n1, op.work.get());
    // bands per K2 CTA: as many as keep about eight CTAs per SM busy
    const int lines = op.n2 * tiles;
    const int groups = std::max(1, std::min(nbc, ceil_div(8 * sms, lines)));
    const int bpc = ceil_div(nbc, groups);
    launch_chained(dim3(lines, ceil_div(nbc, bpc)), xline_threads(op.ax.plan), xsm, s, k2_xlines<R>,
        op.work.get(), op.n1, op.n2, op.n3, op.nplanes, op.slot_plane.get(), op.ax.plan, op.tw.get(), op.veff.get(),
        nbc, bpc);
    launch_chained(dim3(op.nplanes, nbc), pth, psm, s, k3_planes_to_sphere<R>,
        op.work.get(), op.n2, op.n3, op.nplanes, op.plane_start.get(), op.spos.get(), op.row_start.get(),
        op.row_list.get(), op.ay.plan, op.az.plan, op.tw.get() + op.n1, x, ld, b0, op.kinetic.get(), hx, sx);
    pf.launches += 3;
  }
  HALF_LAUNCH("local operator");
  Tuner::finish(tune_token, s, double(nb));
  pf.span(Profile::kLocal, ev_local, pf.record(s));
  {
    // FFT-path algorithmic bytes per band: read psi, write H psi and S psi, two
    // transforms x two passes x (read + write) of the box; Veff once per call.
    const double sz = sizeof(C), rz = sizeof(R), nr = double(op.n1) * op.n2 * op.n3;
    pf.local_bytes += nb * (3.0 * sz * op.npw + 8.0 * sz * nr) + rz * nr;
    pf.local_columns += nb;
  }
  if (op.np > 0) {
    pf.launches += 1;
    apply_nonlocal<R>(rt, op, x, ld, nb, hx, sx);
  }
  pf.span(Profile::kSweep, ev_sweep, pf.record(s));
  pf.sweep_columns += nb;
}

namespace {

// The planes of B given back; the products go to ZGEMM from here on.
void release_integer(KOperator<double>& op) {
  op.integer = false;
  op.crt_bh = op.crt_b = CrtPlanes();
  op.crt_bh_store.release();
  op.crt_b_store.release();
}

}  // namespace

void release_solve_planes(KOperatorSet& ks) {
  if (ks.op64) release_integer(*ks.op64);
}

// Projector part: H X += B blockdiag(D) B^H X, S X += B blockdiag(Q) B^H X
template <typename R>
void apply_nonlocal(Runtime& rt, KOperator<R>& op, const cplx_t<R>* x, long long ld, int nb, cplx_t<R>* hx,
                    cplx_t<R>* sx) {
  using C = cplx_t<R>;
  cudaStream_t s = rt.stream;
  if (op.ws_cols < nb) {
    op.coeff.resize((size_t)op.np * nb);
    op.dy.resize((size_t)op.np * nb);
    op.qy.resize((size_t)op.np * nb);
    op.ws_cols = nb;
  }
  const C one = cval<R>(1.0), zero = cval<R>(0.0);
  auto mix = [&]() {
    launch_chained(ceil_div((long long)op.np * nb, 256), 256, 0, s, mix_kernel<R>,
        op.coeff.get(), op.np, nb, op.col_base.get(), op.col_a.get(), op.col_nlm.get(), op.col_dofs.get(),
        op.col_qofs.get(), op.dall.get(), op.qall.get(), op.dy.get(), op.qy.get());
    HALF_LAUNCH("mix");
    ++rt.prof.launches;
  };
  if constexpr (sizeof(R) == 4) {
    // FP32: B in bf16 planes split once per k point (fill_operator).
    //   coeff = conj(B)^T X            (np x nb, K = npw)
    //   [H X | S X] += B [DY | QY]     (npw x 2nb, K = np; one GEMM, two outputs)
    tc_cgemm(rt, op.bh_planes, tc_dense_b(CUBLAS_OP_N, x, ld, op.npw, nb), op.np, nb, op.npw, make_double2(1, 0),
             make_double2(0, 0), op.coeff.get(), false, op.np);
    mix();
    TcOperand y = tc_dense_b(CUBLAS_OP_N, op.dy.get(), op.np, op.np, 2 * nb);
    y.p2 = op.qy.get();
    y.split = nb;
    tc_cgemm(rt, op.b_planes, y, op.npw, 2 * nb, op.np, make_double2(1, 0), make_double2(1, 0), hx, false, ld, sx, nb);
  } else {
    const bool kept = op.crt_bh.planes != nullptr;
    auto room = [&]() {   // for the planes of B and of the blocks, and the residues
      const size_t block = std::max(crt_plane_bytes(nb, op.npw, true), crt_plane_bytes(2 * nb, op.np, true));
      const size_t result = std::max(crt_result_bytes(rt.sms, op.np, nb, op.npw),
                                     crt_result_bytes(rt.sms, op.npw, 2 * nb, op.np));
      const bool ok = crt_reserve(rt, 0, block, result) &&
                      op.crt_bh_store.try_reserve(crt_plane_bytes(op.np, op.npw, false)) &&
                      op.crt_b_store.try_reserve(crt_plane_bytes(op.npw, op.np, false));
      if (!ok) release_integer(op);
      return ok;
    };
    if (op.integer && zcrt_serves(rt.sms, op.np, nb, op.npw, kept) &&
        zcrt_serves(rt.sms, op.npw, 2 * nb, op.np, kept) && room()) {
      // coeff = B^H X, [H X | S X] += B [DY | QY] on the integer tensor cores
      CrtSide s;
      s.ld = op.npw;
      if (!kept) {
        s.p = op.B.get();
        s.rows = op.np;
        s.k = op.npw;
        s.kcontig = s.conj = true;
        op.crt_bh = crt_prepare(rt, s, false, op.crt_bh_store);
        s.rows = op.npw;
        s.k = op.np;
        s.kcontig = s.conj = false;
        op.crt_b = crt_prepare(rt, s, false, op.crt_b_store);
      }
      s.p = x;
      s.ld = ld;
      s.rows = nb;
      s.k = op.npw;
      s.kcontig = true;
      s.conj = false;
      crt_product(rt, op.crt_bh, crt_prepare(rt, s, true, rt.crt_b), one, zero, op.coeff.get(), op.np);
      mix();
      s.p = op.dy.get();
      s.p2 = op.qy.get();
      s.split = nb;
      s.ld = op.np;
      s.rows = 2 * nb;
      s.k = op.np;
      crt_product(rt, op.crt_b, crt_prepare(rt, s, true, rt.crt_b), one, one, hx, ld, false, sx, nb);
      return;
    }
    gemm(rt, CUBLAS_OP_C, CUBLAS_OP_N, op.np, nb, op.npw, one, op.B.get(), op.npw, x, ld, zero, op.coeff.get(), op.np);
    mix();
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, op.npw, nb, op.np, one, op.B.get(), op.npw, op.dy.get(), op.np, one, hx, ld);
    gemm(rt, CUBLAS_OP_N, CUBLAS_OP_N, op.npw, nb, op.np, one, op.B.get(), op.npw, op.qy.get(), op.np, one, sx, ld);
  }
}

template void apply_hs<double>(Context&, KOperatorSet&, const double2*, long long, int, double2*, double2*, int);
template void apply_hs<float>(Context&, KOperatorSet&, const float2*, long long, int, float2*, float2*, int);

namespace {
template <typename A, typename B>
__global__ void convert_complex_kernel(const A* __restrict__ in, B* __restrict__ out, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) {
    B v;
    v.x = in[i].x;
    v.y = in[i].y;
    out[i] = v;
  }
}
}  // namespace

void apply_hs_fp32(Context& ctx, KOperatorSet& ks, const double2* x, long long n, int nb, double2* hx, double2* sx,
                   int chunk) {
  cudaStream_t s = ks.rt->stream;
  const long long tot = n * nb;
  DeviceBuffer<float2> x32(tot), h32(tot), s32(tot);
  convert_complex_kernel<double2, float2><<<ceil_div(tot, 256), 256, 0, s>>>(x, x32.get(), tot);
  HALF_LAUNCH("to FP32");
  apply_hs<float>(ctx, ks, x32.get(), n, nb, h32.get(), s32.get(), chunk);
  convert_complex_kernel<float2, double2><<<ceil_div(tot, 256), 256, 0, s>>>(h32.get(), hx, tot);
  convert_complex_kernel<float2, double2><<<ceil_div(tot, 256), 256, 0, s>>>(s32.get(), sx, tot);
  HALF_LAUNCH("to FP64");
  HALF_CUDA(cudaStreamSynchronize(s));
}

void accumulate_band_density(KOperatorSet& ks, const double2* x, long long ld, int nb, const double* bw,
                             double* density_c, int chunk) {
  KOperator<double>& op = pick<double>(ks);
  cudaStream_t s = ks.rt->stream;
  if (nb <= 0) return;
  if (chunk <= 0) chunk = 16;
  chunk = std::max(1, std::min(chunk, nb));
  if (op.work_chunk < chunk) {
    op.work.resize((size_t)chunk * op.nplanes * op.n2 * op.n3);
    op.work_chunk = chunk;
  }
  const size_t psm = plane_smem<double>(op.n2, op.n3);
  const int pth = plane_threads<double>(psm);
  const size_t dsm = xline_smem<double>(op.n1);   // its accumulator takes the Veff tile's place
  raise_smem_limit(k2_density, dsm);
  const int tiles = (op.n3 + kXTile - 1) / kXTile;
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    const int nbc = std::min(chunk, nb - b0);
    launch_chained(dim3(op.nplanes, nbc), pth, psm, s, k1_sphere_to_planes<double>,
        x, ld, b0, op.n2, op.n3, op.nplanes, op.plane_start.get(), op.spos.get(), op.row_start.get(),
        op.row_list.get(), op.ay.plan, op.az.plan, op.tw.get() + op.n1, op.work.get());
    k2_density<<<op.n2 * tiles, xline_threads(op.ax.plan), dsm, s>>>(
        op.work.get(), op.n1, op.n2, op.n3, op.nplanes, op.slot_plane.get(), op.ax.plan, op.tw.get(), bw + b0, nbc,
        density_c);
    ks.rt->prof.launches += 2;
  }
  HALF_LAUNCH("band density");
}

// Projector matrix of the prepared k point (used by the dense path and forces).
const double2* projector_matrix64(KOperatorSet& ks) { return pick<double>(ks).B.get(); }

}  // namespace hb
