// The box of quads that a tile's footprint on the detector spans.
#pragma once

#include <cuda_runtime.h>

namespace lct {

__host__ __device__ constexpr int clamp_int(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// corners {row_lo, row_hi, col_lo, col_hi} (rows in quad rows, columns in detector columns, any int: the
// conversion of a corner saturates) -> quad rows and columns {row_lo, row_hi, col_lo, col_hi}, one wider
// on each side, row_lo <= row_hi and col_lo <= col_hi, all inside a view of (nt + 3) x (ns + 3) quads.  Clamped
// before the steps of one and two, so that none can overflow.
__host__ __device__ constexpr int4 box_in_view(const int4& c, int ns, int nt) {
  int4 b = {};
  b.x = clamp_int(c.x, 1, nt + 3) - 1;
  b.y = clamp_int(c.y, b.x - 1, nt + 1) + 1;
  b.z = clamp_int(c.z, -1, ns + 1) + 1;
  b.w = clamp_int(c.w, b.z - 3, ns - 1) + 3;
  return b;
}

}  // namespace lct
