// Plane-wave basis of one k point (src/half_basis.F90:9-55): the box loop
// n1 -> n2 -> n3 over [-n/2, (n-1)/2], kept when hbar^2/2m |k+G|^2 < ENCUT.
// The G order is ABI-visible through half_get_basis and must match exactly.
//
// Along n3 the kinetic energy is a parabola, so each row's kept points lie in
// one interval.  It is found from the parabola's roots, widened by a point on
// either side against rounding, and only inside it is the energy evaluated,
// by the same expression for every point: the whole box took 0.7 ms of host
// time for a 60^3 box with 11,000 kept points.
#include <algorithm>
#include <cmath>

#include "context.h"

namespace hb {

Basis build_basis(const Crystal& c, const std::array<int, 3>& shape, double encut, const double k[3]) {
  if (!(encut > 0)) fail(kInvalidArgument, "ENCUT must be positive");
  Basis b;
  b.shape = shape;
  for (int j = 0; j < 3; ++j) b.kpoint[j] = k[j];
  auto rec = c.reciprocal();
  const int s1 = shape[0], s2 = shape[1], s3 = shape[2];
  const double a2 = rec[6] * rec[6] + rec[7] * rec[7] + rec[8] * rec[8];
  const double lim = encut / kHsqdtm;
  const double box = double(s1) * s2 * s3;
  const double sphere = 1.1 * lim * std::sqrt(lim) * std::fabs(c.volume()) / (6.0 * kPi * kPi) + 64.0;
  const size_t guess = size_t(sphere < box ? sphere : box);
  b.gvec.reserve(3 * guess);
  b.qvec.reserve(3 * guess);
  b.kinetic.reserve(guess);
  b.fft_index.reserve(guess);
  for (int n1 = -(s1 / 2); n1 <= (s1 - 1) / 2; ++n1)
    for (int n2 = -(s2 / 2); n2 <= (s2 - 1) / 2; ++n2) {
      const double f0 = n1 + k[0], f1 = n2 + k[1];
      double base[3];
      for (int j = 0; j < 3; ++j) base[j] = f0 * rec[0 * 3 + j] + f1 * rec[1 * 3 + j];
      // |base + f2 a|^2 < lim around its minimum f2 = -a.base / a.a
      const double mid = -(base[0] * rec[6] + base[1] * rec[7] + base[2] * rec[8]) / a2;
      const double perp = base[0] * base[0] + base[1] * base[1] + base[2] * base[2] - mid * mid * a2;
      const double room = (lim - perp) / a2;
      // A row whose minimum misses the sphere by less than rounding is still looked at.
      if (!(room > -1e-6 * (1.0 + lim / a2))) continue;
      const double half = std::sqrt(std::max(0.0, room)) + 1.01;
      // clamped to the box before the conversion: a k point far away may put the interval outside int
      const double first = -(s3 / 2), last = (s3 - 1) / 2;
      const int lo = int(std::min(std::max(first, std::floor(mid - half - k[2])), last + 1.0));
      const int hi = int(std::max(std::min(last, std::ceil(mid + half - k[2])), first - 1.0));
      for (int n3 = lo; n3 <= hi; ++n3) {
        const double f2 = n3 + k[2];
        double q[3];
        for (int j = 0; j < 3; ++j) q[j] = base[j] + f2 * rec[2 * 3 + j];
        double kin = kHsqdtm * (q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
        if (kin < encut) {
          b.gvec.push_back(n1);
          b.gvec.push_back(n2);
          b.gvec.push_back(n3);
          b.qvec.insert(b.qvec.end(), {q[0], q[1], q[2]});
          b.kinetic.push_back(kin);
          long long i1 = ((n1 % s1) + s1) % s1, i2 = ((n2 % s2) + s2) % s2, i3 = ((n3 % s3) + s3) % s3;
          b.fft_index.push_back((i1 * s2 + i2) * s3 + i3);
        }
      }
    }
  return b;
}

}  // namespace hb
