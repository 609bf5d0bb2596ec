// Scan simulator (no reference counterpart): analytic line integrals of an ellipsoid phantom
// along the helical fan-beam rays of the reference geometry, plus Poisson noise.
//
// Geometry, recovered from the reference kernels (the rebin takes fan view ia + alpha/orbit
// for parallel view ia, CUDA/Rebiner.cu:92-100; the backprojector inverts it with
// theta = asin(phat/dso) and lhat = sqrt(dso^2 - phat^2) + x sin b - y cos b,
// CUDA/Backprojector.cu:53-61):
//   source at angle b, couch z:  S = (-R sin b, R cos b, z)
//   column is:   fan angle a = (is - ws) ds / R (equiangular)
//   in-plane ray direction:      (sin(b - a), -cos(b - a))
//   row it:      iso-scaled height t = (it - wt) dt; the ray rises t / R per unit in-plane length
// Noise: counts ~ Poisson(I0 exp(-p)) drawn from a counter-based Philox4x32-10 stream
// (Salmon et al., SC'11) -- Knuth's product method below 30 expected counts, a rounded
// normal N(l, l) above -- clamped to >= 1, then p = -ln(counts / I0).  The CPU oracle
// evaluates the identical formulas, so GPU and CPU scans agree to rounding.
#include <cmath>

#include "lct_internal.h"

namespace lct {

constexpr int kSimMaxEllipsoids = 128;

__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t lo0 = 0xD2511F53u * c[0], hi0 = __umulhi(0xD2511F53u, c[0]);
    const uint32_t lo1 = 0xCD9E8D57u * c[2], hi1 = __umulhi(0xCD9E8D57u, c[2]);
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ double noisy_integral(double p, double i0, uint64_t seed, uint64_t idx) {
  if (i0 <= 0.0) return p;
  uint32_t c[4] = {(uint32_t)idx, (uint32_t)(idx >> 32), 0x4c435430u, 0u};
  philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double u1 = ((double)c[0] + 0.5) * (1.0 / 4294967296.0);
  const double u2 = ((double)c[1] + 0.5) * (1.0 / 4294967296.0);
  const double lam = i0 * exp(-p);
  double n;
  if (lam < 30.0) {
    const double L = exp(-lam);
    double prod = u1;
    int k = 0, j = 0;
    uint32_t cc[4] = {c[2], c[3], 0x4b4e5554u, 0u};
    while (prod > L && k < 1000) {
      ++k;
      if (j == 4) {
        philox4x32_10(cc, (uint32_t)seed, (uint32_t)(seed >> 32));
        j = 0;
      }
      prod *= ((double)cc[j++] + 0.5) * (1.0 / 4294967296.0);
    }
    n = k;
  } else {
    n = floor(lam + sqrt(lam * (-2.0 * log(u1))) * cospi(2.0 * u2) + 0.5);
  }
  if (n < 1.0) n = 1.0;
  return -log(n * (1.0 / i0));
}

// Bound: the FP64 pipe.  With M = the ellipsoid's frame scaled to a unit sphere, the ray S + l D
// meets it where |M (S - c) + l M D| = 1, a quadratic with coefficients A = |M D|^2, B and C.  D is
// (Dx, Dy) of the column and tz of the row, so A is a quadratic and B a line in tz whose
// coefficients need the column only: a thread makes up to 16 rows of one column and pays, per
// ellipsoid, about 20 operations for the column and 2 per row (the discriminant B^2 - A C, a quadratic
// in the row), where the products with the rotation and six divisions per ray took about 100.  The
// chord sqrt(disc) / A, where there is one, is one rsqrt.
// 600 views x 64 x 736, 40 ellipsoids, I0 = 1e5: 1.1 ms, one ray per thread with everything
// evaluated per ray 8.4 ms.
// A launch that leaves the chip's CTA slots empty is bound by one thread's time instead: it takes ROWS = 4
// rows per thread, or 1.  One view x 16 x 736: 67 us with 16 rows per thread, 20 with 1 (one ray per thread
// with everything evaluated per ray 39).  A row is a step from its 16's first row in any of them, so its
// value does not depend on the launch.
constexpr int kSimRows = 16;     // rows whose quadratics share a base
constexpr int kSimThreads = 128; // columns per CTA
constexpr int kSimCtas = 5;      // CTAs per SM

struct SimEllipsoid {            // one ellipsoid seen from one view
  double xx, xy2, yy, xz2, yz2, zz;  // M^T M, off-diagonal terms doubled
  double bx, by, bz, c;              // (M (S - c)) . M's columns, |M (S - c)|^2 - 1
  double mu2;                        // 2 mu
};

// grid (ceil(ns / 128), row chunks, views); CTA: 128 columns x rows_per_cta rows of one view
template <int ROWS>
__global__ void __launch_bounds__(kSimThreads, kSimCtas) sim_project_kernel(
    const double* __restrict__ ell, int ne, int ns, int nt, int rows_per_cta, float ds, float dt,
    float ws, float wt, float dso, const double* __restrict__ angles,
    const double* __restrict__ zpos, long long v0, double i0, uint64_t seed,
    float* __restrict__ fan) {
  __shared__ SimEllipsoid s_e[kSimMaxEllipsoids];
  const long long v = v0 + blockIdx.z;
  const double R = dso;
  const double b = angles[v];
  if ((int)threadIdx.x < ne) {  // ne <= kSimMaxEllipsoids = kSimThreads
    const double* e = ell + 16 * threadIdx.x;  // cx cy cz ax ay az rot[9] mu
    double sb, cb;
    sincos(b, &sb, &cb);
    const double q[3] = {-R * sb - e[0], R * cb - e[1], zpos[v] - e[2]};
    SimEllipsoid o = {0, 0, 0, 0, 0, 0, 0, 0, 0, -1.0, 2.0 * e[15]};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double ia = 1.0 / e[3 + r];
      const double mx = e[6 + r] * ia, my = e[9 + r] * ia, mz = e[12 + r] * ia;
      const double sv = mx * q[0] + my * q[1] + mz * q[2];
      o.xx += mx * mx;
      o.xy2 += 2.0 * mx * my;
      o.yy += my * my;
      o.xz2 += 2.0 * mx * mz;
      o.yz2 += 2.0 * my * mz;
      o.zz += mz * mz;
      o.bx += sv * mx;
      o.by += sv * my;
      o.bz += sv * mz;
      o.c += sv * sv;
    }
    s_e[threadIdx.x] = o;
  }
  __syncthreads();
  const int is = blockIdx.x * kSimThreads + threadIdx.x;
  if (is >= ns) return;
  const double a = ((double)is - ws) * ds / R;
  double dx, dy;
  sincos(b - a, &dx, &dy);
  dy = -dy;
  const double dxx = dx * dx, dxy = dx * dy, dyy = dy * dy;
  const double step = (double)dt / R;  // tz from one row to the next
  const int row1 = min(nt, (int)(blockIdx.y + 1) * rows_per_cta);
  for (int it0 = blockIdx.y * rows_per_cta; it0 < row1; it0 += ROWS) {
    const int base = it0 / kSimRows * kSimRows;
    const double t0 = ((double)base - wt) * dt / R;
    const double r0 = ROWS == kSimRows ? 0.0 : (double)(it0 - base);  // steps from the base to the first row
    const unsigned rows = (1u << min(ROWS, row1 - it0)) - 1u;         // of this pass
    double p[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) p[r] = 0.0;
    for (int m = 0; m < ne; ++m) {
      const SimEllipsoid& e = s_e[m];
      // A and B at row base + r: A0 + r (A1 + r A2), B0 + r B1; the discriminant B^2 - A c is a
      // quadratic in r too, and A is needed where it is positive only
      const double ul = fma(dx, e.xz2, dy * e.yz2), tl = fma(t0, e.zz, ul);
      const double A0 = fma(t0, tl, fma(dxx, e.xx, fma(dxy, e.xy2, dyy * e.yy)));
      const double A1 = step * fma(t0, e.zz, tl), A2 = step * step * e.zz;
      const double B0 = fma(t0, e.bz, fma(dx, e.bx, dy * e.by)), B1 = step * e.bz;
      const double c = e.c, mu2 = e.mu2;
      const double d0 = fma(B0, B0, -(A0 * c)), d1 = fma(2.0 * B0, B1, -(A1 * c)), d2 = fma(B1, B1, -(A2 * c));
      unsigned hit = 0;
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (fma(r0 + r, fma(r0 + r, d2, d1), d0) > 0.0) hit |= 1u << r;
      hit &= rows;
      if (!hit) continue;
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if ((hit >> r) & 1u) {
          const double disc = fma(r0 + r, fma(r0 + r, d2, d1), d0);
          const double A = fma(r0 + r, fma(r0 + r, A2, A1), A0);
          p[r] = fma(mu2 * disc, rsqrt(disc * A * A), p[r]);  // sqrt(disc) / A
        }
    }
#pragma unroll 2
    for (int r = 0; r < ROWS; ++r) {
      const int it = it0 + r;
      if (it >= row1) break;
      double pr = p[0];
#pragma unroll
      for (int k = 1; k < ROWS; ++k) pr = r == k ? p[k] : pr;
      const double tz = ((double)it - wt) * dt / R;
      const uint64_t idx = ((uint64_t)v * nt + it) * ns + is;
      fan[((long long)blockIdx.z * nt + it) * ns + is] =
          (float)noisy_integral(pr * sqrt(1.0 + tz * tz), i0, seed, idx);
    }
  }
}

// voxelised phantom: one thread per voxel, ss^3 sub-samples, ellipsoids in shared memory
__global__ void __launch_bounds__(128) voxelise_kernel(const double* __restrict__ ell, int ne,
                                                       int nx, int ny, double x0, double y0,
                                                       double z0, double dx, double dy,
                                                       double dz, int ss, float* __restrict__ out) {
  __shared__ double s_e[kSimMaxEllipsoids * 16];
  for (int i = threadIdx.x; i < ne * 16; i += blockDim.x) s_e[i] = ell[i];
  __syncthreads();
  const int ix = blockIdx.x * blockDim.x + threadIdx.x;
  const int iy = blockIdx.y, iz = blockIdx.z;
  if (ix >= nx) return;
  double acc = 0.0;
  for (int sz = 0; sz < ss; ++sz)
    for (int sy = 0; sy < ss; ++sy)
      for (int sx = 0; sx < ss; ++sx) {
        const double P[3] = {x0 + (ix + (sx + 0.5) / ss - 0.5) * dx,
                             y0 + (iy + (sy + 0.5) / ss - 0.5) * dy,
                             z0 + (iz + (sz + 0.5) / ss - 0.5) * dz};
        for (int m = 0; m < ne; ++m) {
          const double* e = s_e + 16 * m;
          const double* R = e + 6;
          const double p[3] = {P[0] - e[0], P[1] - e[1], P[2] - e[2]};
          const double u0 = (R[0] * p[0] + R[3] * p[1] + R[6] * p[2]) / e[3];
          const double u1 = (R[1] * p[0] + R[4] * p[1] + R[7] * p[2]) / e[4];
          const double u2 = (R[2] * p[0] + R[5] * p[1] + R[8] * p[2]) / e[5];
          if (u0 * u0 + u1 * u1 + u2 * u2 <= 1.0) acc += e[15];
        }
      }
  out[((long long)iz * ny + iy) * nx + ix] = (float)(acc / ((double)ss * ss * ss));
}

}  // namespace lct

using namespace lct;

LCT_API int lct_voxelise(const double* d_ellipsoids, int n_ellipsoids, int nx, int ny, int nz,
                         double x0, double y0, double z0, double dx, double dy, double dz, int ss,
                         float* d_out, lct_stream stream) {
  if (!d_ellipsoids || n_ellipsoids < 0 || n_ellipsoids > kSimMaxEllipsoids || !d_out) return LCT_ERR_ARG;
  if (nx <= 0 || ny <= 0 || nz <= 0 || ny > 65535 || nz > 65535 || ss <= 0 || ss > 16) return LCT_ERR_ARG;
  dim3 grid((nx + 127) / 128, ny, nz);
  voxelise_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(d_ellipsoids, n_ellipsoids, nx, ny, x0,
                                                          y0, z0, dx, dy, dz, ss, d_out);
  return launch_status();
}

LCT_API int lct_sim_project(const double* d_ellipsoids, int n_ellipsoids, int ns, int nt,
                            float ds, float dt, float ws, float wt, float dso,
                            const double* d_angles, const double* d_zpos, int64_t v0, int64_t v1,
                            double i0, uint64_t seed, float* d_fan, lct_stream stream) {
  if (!d_ellipsoids || n_ellipsoids < 0 || n_ellipsoids > kSimMaxEllipsoids) return LCT_ERR_ARG;
  if (ns <= 0 || nt <= 0 || !d_angles || !d_zpos || !d_fan || v1 < v0 || v0 < 0) return LCT_ERR_ARG;
  if (!(ds > 0.f) || !(dt > 0.f) || !(dso > 0.f)) return LCT_ERR_ARG;
  const long long nv = v1 - v0;
  cudaStream_t s = (cudaStream_t)stream;
  // a CTA makes all rows of its columns (the ellipsoids' view terms once) unless that leaves fewer
  // CTAs than 8 per SM; then one pass of rows each, and of as few rows as one round of CTA slots holds
  const int sms = device_sms();
  const int cols = (ns + kSimThreads - 1) / kSimThreads;
  const long long slots = (long long)kSimCtas * sms;
  const int rows = cols * nv * nt <= slots ? 1 : (cols * nv * ((nt + 3) / 4) <= slots ? 4 : kSimRows);
  const int passes = (nt + rows - 1) / rows;
  const int chunks = cols * nv >= 8LL * sms ? (passes + 15) / 16 : passes;
  const int rows_per_cta = (passes + chunks - 1) / chunks * rows;
  const unsigned gy = (unsigned)((nt + rows_per_cta - 1) / rows_per_cta);
  if (gy > 65535) return LCT_ERR_ARG;
  auto kernel = rows == 1 ? sim_project_kernel<1> : (rows == 4 ? sim_project_kernel<4> : sim_project_kernel<kSimRows>);
  for (long long c = 0; c < nv; c += 65535) {
    const long long cnt = nv - c < 65535 ? nv - c : 65535;
    dim3 grid(cols, gy, (unsigned)cnt);
    kernel<<<grid, kSimThreads, 0, s>>>(d_ellipsoids, n_ellipsoids, ns, nt, rows_per_cta, ds, dt, ws, wt, dso,
                                        d_angles, d_zpos, v0 + c, i0, seed, d_fan + c * (long long)nt * ns);
    int st = launch_status();
    if (st) return st;
  }
  return LCT_OK;
}
