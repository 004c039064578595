// Complex FP64 products on the integer tensor cores (zcrt.cu).
#pragma once

#include "context.h"

namespace hb {

// An operand: op(A) as rows r over k, or op(B) as its columns r over k.
// Element (r, k) at p[k + r ld] when k is contiguous, else at p[r + k ld];
// rows (k contiguous) or k (otherwise) from `split` on continue at p2.
struct CrtSide {
  const double2* p = nullptr;
  const double2* p2 = nullptr;
  int split = INT32_MAX;
  long long ld = 0;
  int rows = 0, k = 0;
  bool kcontig = false, conj = false;
};

// The residue planes of an operand and its rows' scales.
struct CrtPlanes {
  const unsigned char* planes = nullptr;
  const int* e = nullptr;
  int rows = 0, rows_pad = 0, k = 0, k_pad = 0;
};

// Splits an operand into `store` (resized when too small); `as_b`: the
// right-hand operand of products, else the left-hand one.
CrtPlanes crt_prepare(Runtime& rt, const CrtSide& s, bool as_b, DeviceBuffer<unsigned char>& store);

// Bytes of an operand's planes, and of the residues of an m x n product over k.
size_t crt_plane_bytes(int rows, int k, bool as_b);
size_t crt_result_bytes(int sms, int m, int n, int k);

// The runtime's buffers grown to these sizes; false where memory does not
// suffice (the product then goes to ZGEMM).
bool crt_reserve(Runtime& rt, size_t a, size_t b, size_t result);

// C (a.rows x b.rows, ldc) = alpha A B + beta C; columns from split_col on go
// to C2 (column 0 on).  upper: tiles below the diagonal are left out.
void crt_product(Runtime& rt, const CrtPlanes& a, const CrtPlanes& b, double2 alpha, double2 beta, double2* C,
                 long long ldc, bool upper = false, double2* C2 = nullptr, int split_col = INT32_MAX);

// Whether an m x n product over k is large enough to gain over ZGEMM (a_kept:
// the left operand's planes exist already) and within the method's range and
// memory.
bool zcrt_serves(int sms, int m, int n, int k, bool a_kept = false);

}  // namespace hb
