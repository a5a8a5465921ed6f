// gi_record.h -- where a march record keeps its values (MarchArgs::rec_hc, rec_mask,
// rec_hc0): plain C++, used by the kernels, the launches and host programs.
//
// All offsets are 64-bit: a record holds fewer than 2^31 pixels (checked at launch), but
// 64 rows of them are up to 2^37 values (rows of 2^32 values and more start at 9216 x
// 8192 with 58 steps).
#pragma once

#include <stddef.h>

#if defined(__CUDACC__)
#define GI_RECORD_HD __host__ __device__ __forceinline__
#else
#define GI_RECORD_HD static inline
#endif

namespace gi {

// Pixels of a record: every (pattern, sub-image pixel) slot, P^2 ceil(W/P) ceil(H/P).
GI_RECORD_HD size_t record_pixels(int width, int height, int pattern) {
  const size_t P = (size_t)pattern;
  return P * P * (((size_t)width + P - 1) / P) * (((size_t)height + P - 1) / P);
}

// First value of direction d's block of rec_hc (`steps` rows of `npix` values), and of
// row `step` within a block.
GI_RECORD_HD size_t record_block(int d, int steps, unsigned npix) { return (size_t)d * (size_t)steps * npix; }
GI_RECORD_HD size_t record_row(int step, unsigned npix) { return (size_t)(unsigned)step * npix; }

}  // namespace gi
