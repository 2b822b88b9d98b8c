// Reciprocals and reciprocal square roots from the hardware's estimates, each
// refined by a named method, with the errors that the tests hold them to.
#pragma once

namespace bem {
namespace {

// 1 / sqrt(x) for positive normal x: the hardware's estimate y (rsqrt.approx)
// and the first two terms of the binomial series of 1 / sqrt(x) =
// y (1 - e)^(-1/2) with e = 1 - x y^2, y + y e (1/2 + 3/8 e), which take an error
// of 2^-19 below that of the roundings: within 2 ulp.  0, subnormal and infinite
// x give NaN: the callers keep them out.
__device__ __forceinline__ double rsqrt_pos(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1 / a, a != 0, by quotients of a scaled by the power of two of its larger part
// (out of line: 1% of an 800-panel sweep, in line 2.5%).
__device__ __noinline__ double2 cinv(double2 a) {
  const int e = ilogb(fmax(fabs(a.x), fabs(a.y)));
  const double x = scalbn(a.x, -e), y = scalbn(a.y, -e), n = x * x + y * y;
  return make_double2(scalbn(x / n, -e), scalbn(-y / n, -e));
}
// The same without a branch where the square of the modulus is well inside the
// range of float64: the hardware's estimate of the reciprocal and two steps of
// Newton-Raphson for 1 / d, r + r (1 - d r).  Both within 4 x 2^-53 in each part.
__device__ __forceinline__ double2 cinv_fast(double2 a, bool& in_range) {
  const double d = a.x * a.x + a.y * a.y;
  in_range = d > 1e-280 && d < 1e280;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  return make_double2(a.x * r, -a.y * r);
}

// 1 / (re + i im) in float32 for any pivot: where the square of its modulus is far
// inside the range of float32, conj(pivot) times the hardware's estimate of 1 / d
// (rcp.approx, which flushes) and one step of Newton-Raphson for 1 / d,
// r + r (1 - d r); elsewhere quotients of the pivot scaled by the power of two of
// its larger part (out of line: the range costs 2 us per block, in line 3).  Both
// within 4 x 2^-24 in each part.  0 for a zero pivot, infinite for one below 2^-128.
__device__ __noinline__ float2 gj_reciprocal_scaled(float re, float im) {
  const float m = fmaxf(fabsf(re), fabsf(im));
  if (!(m > 0.0f)) return make_float2(0.0f, 0.0f);
  const int e = ilogbf(m);
  const float x = scalbnf(re, -e), y = scalbnf(im, -e), n = x * x + y * y;
  return make_float2(scalbnf(x / n, -e), scalbnf(-y / n, -e));
}
__device__ __forceinline__ float2 gj_reciprocal(float re, float im) {
  const float d = re * re + im * im;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-d, r, 1.0f), r);
  float2 out = make_float2(re * r, -im * r);
  // the pivot is the same in every lane: no divergence
  if (!(d > 0x1p-100f && d < 0x1p100f)) out = gj_reciprocal_scaled(re, im);
  return out;
}

}  // namespace
}  // namespace bem
