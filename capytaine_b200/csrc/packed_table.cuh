// The tabulation of the Delhommeau integrals packed for the pair kernels, and
// its lookup.
//
// The plain table holds the five integrals of a node in 40 bytes, so that the
// 3 x 3 stencil of a lookup is 45 loads of 8 bytes per thread (and 12 more for
// the grid values and the reciprocal Lagrange denominators): with every lane
// on its own node the load pipe, not the float64 pipe, set the speed of the
// wave term.  A variant of the Green function only needs four of the five
// integrals (I0 or I1, and I2, I3, I4), which make one aligned 32-byte quad:
// nine 256-bit loads per lookup, and one per grid for the stencil's record.
//
// Layout, in doubles (the buffer 32-byte aligned):
//   [0, 16)             grid constants: r of the last node, |z| of the last
//                       node, log step of the scaled z grid, slope of the
//                       linear part of the scaled r grid, its node of r = 1
//   4 nr                r stencils (packed_weights)
//   4 nz                z stencils
//   4 nr nz             (I0, I2, I3, I4): the low_freq variant
//   4 nr nz             (I1, I2, I3, I4): the high_freq variant
#pragma once
#include "common.cuh"

namespace bem {

constexpr int kPackHeader = 16;
inline int64_t packed_table_doubles(int nr, int nz) {
  return kPackHeader + 4 * ((int64_t)nr + nz) + 8 * (int64_t)nr * nz;
}

#ifdef __CUDACC__
namespace {

__device__ __forceinline__ void ldg256(const double* p, double& a, double& b, double& c, double& d) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

struct PackedTab {
  const double* base;   // NULL: no packed table
  int nr, nz, grid;
  // read from the header by load()
  const double* r_rec;
  const double* z_rec;
  const double* quads;
  double rmax, zmax, dz, r_slope;
  float r_slope_f, one_f, log_scale_f, inv_dz_f;
  int one;

  __device__ __forceinline__ void load(bool high) {
    rmax = __ldg(base);
    zmax = __ldg(base + 1);
    dz = __ldg(base + 2);
    r_slope = __ldg(base + 3);
    one = (int)__ldg(base + 4);
    r_slope_f = (float)r_slope;
    one_f = (float)one;
    log_scale_f = 0.1f * (one_f - 1.0f);
    inv_dz_f = 1.0f / (float)dz;
    r_rec = base + kPackHeader;
    z_rec = r_rec + 4 * nr;
    quads = z_rec + 4 * nz + (high ? (size_t)4 * nr * nz : 0);
  }
};

// q rounded half away from zero when q (a float32 estimate) is more than
// margin away from every rounding boundary; the caller decides with the
// float64 expression otherwise.
__device__ __forceinline__ bool nint_clear_f(float q, float margin, int& out) {
  const float fl = floorf(q);
  const float fr = q - fl;
  out = (int)fl + (fr > 0.5f ? 1 : 0);
  return fabsf(fr - 0.5f) > margin;
}
__device__ __forceinline__ float log10_approx(float x) { return 0.30102999566f * __log2f(x); }

// Nodes of Delhommeau_integrals.f90:301-363 on the scaled grid from float32
// estimates of the same expressions.  __log2f errs by 2^-22 relative, i.e. by
// 2.4e-6 in log10 down to 1e-10; with the roundings of the float32 arithmetic
// the estimate is within 5e-6 (log10 units) or 3e-7 of the terms' magnitude,
// and the margins are twice that.  Within a margin the float64 expressions
// decide, so the node is always theirs.
template <class Exact>
__device__ __forceinline__ int packed_r_node(double r, const PackedTab& P, Exact&& exact) {
  int i;
  const float rf = (float)r;
  float q, margin;
  if (rf < 1.0f) {
    q = fmaxf(fmaf(log10_approx(rf), P.log_scale_f, P.one_f), 0.0f);
    margin = 1e-5f * P.one_f;
  } else {
    q = fmaf(rf - 1.0f, P.r_slope_f, P.one_f);
    margin = 6e-7f * fmaf(rf, P.r_slope_f, P.one_f);
  }
  if (P.grid == kLegacyGrid || !nint_clear_f(q, margin, i)) i = exact(r);
  return max(2, min(P.nr - 1, i));
}
template <class Exact>
__device__ __forceinline__ int packed_z_node(double z, const PackedTab& P, Exact&& exact) {
  int j;
  const float q = fmaxf((log10_approx(fabsf((float)z)) + 10.0f) * P.inv_dz_f, 0.0f);
  if (P.grid == kLegacyGrid || !nint_clear_f(q, 1e-5f * P.inv_dz_f, j)) j = exact(z);
  return max(2, min(P.nz - 1, j));
}

// Lagrange weights of the three nodes at x from their record (u, 1/b, rho,
// 1/(rho (1 + rho))) with u the middle node, a and b the steps below and above
// it and rho = a/b: with s = (x - u)/b, w0 = s (s - 1)/(rho (1 + rho)), and the
// other two follow from sum w = 1 and sum w u = x.  One load instead of the two
// that nodes and denominators need, and two operations less.
__device__ __forceinline__ void packed_weights(const double* rec, double x, double w[3]) {
  double u, inv_b, rho, kappa;
  ldg256(rec, u, inv_b, rho, kappa);
  const double s = (x - u) * inv_b;
  w[0] = fma(s, s, -s) * kappa;
  w[2] = fma(rho, w[0], s);
  w[1] = (1.0 - w[0]) - w[2];
}

// The four integrals of the variant at (r, z) inside the table (nodes i, j,
// 1-based; wr: the weights of r at node i).
__device__ __forceinline__ void packed_interpolate(const double wr[3], double z, int i, int j, const PackedTab& P,
                                                   double out[4]) {
  double wz[3];
  packed_weights(P.z_rec + 4 * (j - 1), z, wz);
  const double* q = P.quads + 4 * ((size_t)(i - 2) * P.nz + (j - 2));
  out[0] = out[1] = out[2] = out[3] = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double t[3][4];
#pragma unroll
    for (int b = 0; b < 3; ++b) ldg256(q + 4 * b, t[b][0], t[b][1], t[b][2], t[b][3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = fma(wr[a], fma(t[2][k], wz[2], fma(t[1][k], wz[1], t[0][k] * wz[0])), out[k]);
    q += 4 * P.nz;
  }
}

}  // namespace
#endif

}  // namespace bem
