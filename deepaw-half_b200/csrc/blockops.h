// FP64 products of the acc iteration's band blocks (blockops.cu).
//
// A block is n x cols, column-major with leading dimension n, and may be two
// buffers side by side: columns [0, c1) at p1, [c1, c1 + c2) at p2.
#pragma once

#include "context.h"

namespace hb {

struct ZBlock {
  const double2* p1 = nullptr;
  int c1 = 0;
  const double2* p2 = nullptr;
  int c2 = 0;
  int cols() const { return c1 + c2; }
};

// Where a product of blocks runs: small ones on the kernels of blockops.cu,
// large ones on the integer tensor cores (zcrt.cu) where the caller allows
// that, every other on ZGEMM.
enum class ZRoute { kBlock = 1, kInteger = 2, kLibrary = 3 };
ZRoute zgram_route(int sms, int n, int rows, int cols, bool integer);     // A^H B: rows x cols over n
ZRoute zupdate_route(int sms, int n, int k, int cols, bool integer);      // Z Y: n x cols over k

// C_i = A^H B_i for i < count (count 1 or 2, blocks of one shape), written
// with leading dimension ldc.  upper: only the upper triangle is needed (A
// and B_i of equal width and split); elements below it may or may not be written.
void zgram(Runtime& rt, int n, const ZBlock& a, const ZBlock* b, double2* const* c, int count, int ldc, bool upper,
           ZRoute route);

// C_i = beta C_i + alpha Z_i Y for i < count (up to 3 blocks of one shape):
// Z_i n x K, Y K x cols (leading dimension ldy), C_i n x cols, beta 0 or 1.
// C_i overlaps no Z_i.
void zupdate(Runtime& rt, int n, const ZBlock* z, const double2* y, int ldy, double2* const* c, int cols, int count,
             double alpha, double beta, ZRoute route);

}  // namespace hb
