// Copies of band blocks between pageable host memory and the device
// (staging.cpp).
#pragma once

#include "common.h"

namespace hb {

// dst (device, n x cols packed) = src (host, leading dimension ld >= n).  On
// return src has been read; the device side is ordered on s.
void block_to_device(double2* dst, const void* src, long long ld, long long n, long long cols, cudaStream_t s);

// dst (host, leading dimension ld >= n) = src (device, n x cols packed), after
// the work already on s.  On return dst is complete.
void block_to_host(void* dst, long long ld, const double2* src, long long n, long long cols, cudaStream_t s);

// Gives the pinned buffers of the calling process back (last context gone).
void staging_release();

}  // namespace hb
