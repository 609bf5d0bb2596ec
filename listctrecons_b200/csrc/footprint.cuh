// Where samples lie on the detector: the box of quads that a tile's footprint spans, and the test that lets
// a thread read its samples' rows without clamping them.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

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

// Slices j in [jf, jl] of a view have qhat = fma(j, K, M) rows from the detector's centre row and (EXACT)
// the row coordinate fma(j, K, RN(M + wt + 2)).  True where every slice lies within the detector rows, so
// that floor of the coordinate needs no clamp: qhat is monotone in j (a monotone rounding of a linear
// function), so the ends bound it, and the coordinate equals qhat + wt + 2 within a few ulps as long as M is
// not far larger than both.  Two ends on the detector bound K, and with it M; SINGLE (jf = jl, one slice per
// thread) has to bound K itself: next to the source K and M are without bound and may cancel in qhat while
// M + wt + 2 is rounded to many rows.  A NaN is not inside.
template <bool SINGLE>
__host__ __device__ inline bool rows_inside(float jf, float jl, float K, float M, float wt) {
  const bool ends = fabsf(fmaf(jf, K, M)) <= wt && fabsf(fmaf(jl, K, M)) <= wt;
  return SINGLE ? ends && fabsf(K) <= wt + wt : ends;
}

}  // namespace lct
