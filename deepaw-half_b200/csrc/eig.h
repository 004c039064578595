// Device-resident small Hermitian eigensolvers (see eig.cu).
#pragma once

#include <string>
#include <vector>

#include "context.h"

namespace hb {

// Status of a pencil whose grid-wide kernel gave up waiting for its other CTAs.
constexpr int kWaitGaveUp = -100;

// For tests: runtimes that have not asked the device yet take at most clusters
// of this size, and no grid-wide launch unless grid (16, true: the device's own limits).
void limit_pencil_launches(int cluster_ctas, bool grid);

// What went wrong in a solver iteration, from its three status words (metric,
// pencil, factor of the overlap); empty when nothing did.
std::string pencil_failure(const int* infos);

struct SmallEigen {
  // Orders the cluster kernels serve: the matrix fits the shared memory of 16
  // CTAs (432 x 432 x 16 bytes and the vectors).
  static constexpr int kOwnMaxOrder = 432;
  // Orders whose factor and tridiagonalisation go over the whole GPU's shared
  // memory (five rows a thread; 148 SMs hold ceil(n / 148) n elements of 16
  // bytes each up to 1,436).  Above it cuSOLVER.
  static constexpr int kGridMaxOrder = 1280;
  int cap = 0;
  DeviceBuffer<double> d, e, Z, scratch, lam;
  DeviceBuffer<double2> tau, V, work;
  DeviceBuffer<double2> panels;   // exchange buffer of the metric factor's CTAs
  DeviceBuffer<double2> exchange; // and of the grid-wide tridiagonalisation's
  DeviceBuffer<int> grid_state;   // barrier counter and error flag of the grid-wide kernels
  DeviceBuffer<int> info;   // zhetrd status (reports illegal arguments only)
  void reserve(Runtime& rt, int nmax);
  // A (n x n, upper triangle, destroyed) -> nev lowest eigenpairs; vectors in
  // V[:, :nev].  *status (device) becomes nonzero if inverse iteration failed.
  // Where *failed (device; null: never) is nonzero the matrix is of no use, and
  // no eigenvectors are computed.
  void heev(Runtime& rt, double2* A, int n, int nev, double* w, int* status, const int* failed = nullptr);
  // A y = lambda B y, B Hermitian positive definite; Y^H B Y = I.
  // *chol_status (device): nonzero when the factor saw a pivot that is not
  // finite (beyond the grid-wide kernels' orders zpotrf's info).  strict: a
  // pivot that is not positive is an error, as in zpotrf; otherwise dependent
  // and negative pivots are floored as in the metric.
  void hegv(Runtime& rt, double2* A, double2* B, int n, int nev, double* w, int* status, int* chol_status,
            bool strict = false);
  // ACC correction metric: M = P^H S P (m x m) -> U, upper triangular, with
  // (P U)^H S (P U) = I; returns false (nothing launched) when m is not a cluster_order.
  bool metric_normalize(Runtime& rt, double2* M, int m, int* status, bool strict = false);
  // Whether order n goes through the cluster kernels, or above kOwnMaxOrder
  // through the grid-wide ones, whose metric factor floors dependent pivots like
  // the cluster kernel's.  Where the device (or the part of it that the process
  // may use) cannot hold such a launch, neither does, and the order is cuSOLVER's.
  static bool cluster_order(Runtime& rt, int n);
  static bool grid_order(Runtime& rt, int n);

 private:
  void clear_grid_state(cudaStream_t s);
};

// Selected eigenvalues of a large Hermitian matrix A (n x n, column-major,
// upper triangle used and destroyed): Householder tridiagonalisation
// (cuSOLVER zhetrd), then multisection on Sturm counts for the index ranges
// [k0s[r], k0s[r] + counts[r]), written one range after another to lam
// (device).  Synchronises the stream.
void hermitian_eigenvalues_large(Runtime& rt, double2* A, long long n, const std::vector<int>& k0s,
                                 const std::vector<int>& counts, double* lam);

}  // namespace hb
