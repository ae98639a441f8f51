// Phase helpers.  FP32, for the FP32C kernels, that keep work off the SFU/conversion (XU) pipe:
// rounding to an integer by adding and subtracting a power-of-two constant (FP64 or FP32 add
// pipe), and sin/cos of pi x by polynomials on the FMA pipe.  FP64: sin/cos of phases in turns.
#pragma once

#include <cuda_runtime.h>

namespace hgx {

// Round to the nearest integer (ties to even) on the FP64 add pipe, for |x| < 2^51: adding
// 1.5 * 2^52 leaves no fraction bits, subtracting it again returns the rounded value.
constexpr double RND52 = 6755399441055744.0;
__device__ __forceinline__ double round_fp64(double x) { return __dsub_rn(__dadd_rn(x, RND52), RND52); }
// The same in FP32 for |x| < 2^22 (1.5 * 2^23).
__device__ __forceinline__ float round_fp32(float x) { return __fsub_rn(__fadd_rn(x, 12582912.0f), 12582912.0f); }

// sin(pi x) and cos(pi x) for |x| <= 1 in FP32 on the FMA pipe: x = r + k/2 with k = rint(2x)
// (rounded by the 1.5 * 2^23 constant, whose low mantissa bits then hold k mod 4) and
// |r| <= 1/4 exact; Taylor polynomials of sin(pi r)/r (to r^8) and cos(pi r) (to r^10), whose
// truncation is below 2e-9 at |pi r| = pi/4; then the rotation by k quarter turns.  Absolute
// error about one FP32 ulp; sin keeps its relative accuracy near 0.
__device__ __forceinline__ void sincospi_f32(float x, float* s, float* c) {
  const float M = 12582912.0f;
  const float b = __fadd_rn(2.0f * x, M);
  const int q = __float_as_int(b) & 3;
  const float r = x - 0.5f * __fsub_rn(b, M);
  const float r2 = r * r;
  const float ps = fmaf(fmaf(fmaf(fmaf(0.08214588463306427f, r2, -0.5992645025253296f), r2,
                                  2.550163984298706f), r2, -5.167712688446045f), r2,
                        3.1415927410125732f);
  const float pc = fmaf(fmaf(fmaf(fmaf(fmaf(-0.025806890800595284f, r2, 0.23533062636852264f), r2,
                                       -1.3352627754211426f), r2, 4.058712005615234f), r2,
                             -4.934802055358887f), r2, 1.0f);
  const float sv = r * ps;
  float so = (q & 1) ? pc : sv, co = (q & 1) ? -sv : pc;
  if (q & 2) {
    so = -so;
    co = -co;
  }
  *s = so;
  *c = co;
}

// The same for two numbers, two to an FP32x2 operation.
__device__ __forceinline__ void sincospi_f32x2(float2 x, float2* s, float2* c) {
  auto two = [](float v) { return make_float2(v, v); };
  const float2 b = __ffma2_rn(two(2.0f), x, two(12582912.0f));
  const float2 r = __ffma2_rn(two(-0.5f), __fadd2_rn(b, two(-12582912.0f)), x), r2 = __fmul2_rn(r, r);
  float2 ps = __ffma2_rn(two(0.08214588463306427f), r2, two(-0.5992645025253296f));
  ps = __ffma2_rn(ps, r2, two(2.550163984298706f));
  ps = __ffma2_rn(ps, r2, two(-5.167712688446045f));
  ps = __ffma2_rn(ps, r2, two(3.1415927410125732f));
  float2 pc = __ffma2_rn(two(-0.025806890800595284f), r2, two(0.23533062636852264f));
  pc = __ffma2_rn(pc, r2, two(-1.3352627754211426f));
  pc = __ffma2_rn(pc, r2, two(4.058712005615234f));
  pc = __ffma2_rn(pc, r2, two(-4.934802055358887f));
  pc = __ffma2_rn(pc, r2, two(1.0f));
  const float2 sv = __fmul2_rn(r, ps);
  // quarter q: sin takes its sign from bit 1 of q, cos from bit 1 of q + 1
  auto turn = [](float bq, float sn, float cs, float* so, float* co) {
    const unsigned q = __float_as_uint(bq);
    *so = __uint_as_float(__float_as_uint(q & 1 ? cs : sn) ^ ((q & 2) << 30));
    *co = __uint_as_float(__float_as_uint(q & 1 ? sn : cs) ^ (((q + 1) & 2) << 30));
  };
  turn(b.x, sv.x, pc.x, &s->x, &c->x);
  turn(b.y, sv.y, pc.y, &s->y, &c->y);
}

// sin(pi x) for |x| <= 1/2 in FP32: x pi + x (pi's rest + a polynomial of degree 3 in x^2 times x^2, a
// Chebyshev fit), so that the leading product is rounded once, in the sum (within 1.5e-7 of the value, relative
// near 0, 2.8e-8 rms; x times a polynomial: 4.6e-8 rms).
__device__ __forceinline__ float sin_half_turn(float x) {
  const float z = x * x;
  float p = fmaf(0.07854147255420685f, z, -0.598705530166626f);
  p = fmaf(p, z, 2.550136089324951f);
  p = fmaf(p, z, -5.167712688446045f);
  p = fmaf(p, z, -8.742277657347586e-08f);
  return fmaf(x, 3.1415927410125732f, p * x);
}

// sin and cos of 2 pi (r + k/4), |r| <= 1/8: sin(2 pi r) / r and (cos(2 pi r) - 1) / r^2 as polynomials of
// degree 6 in r^2 (Chebyshev fits over the interval; both within 1.4e-16 of the value), k's quarter turns.
__device__ __forceinline__ void sincos_quarters(double r, int k, double* s, double* c) {
  const double z = r * r;
  double p = 3.780830078125, q = -1.698876953125;
  p = fma(p, z, -15.093802528381348);
  q = fma(q, z, 7.9031996917724605);
  p = fma(p, z, 42.05868499483913);
  q = fma(q, z, -26.426253155618905);
  p = fma(p, z, -76.70585970413173);
  q = fma(q, z, 60.24464135185001);
  p = fma(p, z, 81.60524927594797);
  q = fma(q, z, -85.45681720664174);
  p = fma(p, z, -41.341702240399634);
  q = fma(q, z, 64.93939402266824);
  p = fma(p, z, 6.283185307179586);
  q = fma(q, z, -19.739208802178716);
  p *= r;
  q = fma(q, z, 1.0);
  const bool odd = k & 1;
  const double a = odd ? q : p, b = odd ? p : q;
  *s = __hiloint2double(__double2hiint(a) ^ ((k & 2) << 30), __double2loint(a));
  *c = __hiloint2double(__double2hiint(b) ^ (((k + 1) & 2) << 30), __double2loint(b));
}
// sin and cos of 2 pi u in FP64: u reduced exactly by the nearest quarter turn (adding 1.5 2^52 leaves it in
// the low mantissa bits).  18 FP64 operations.  Valid for |u| < 2^50; NaN and infinite u give NaN.
__device__ __forceinline__ void sincos_turns(double u, double* s, double* c) {
  const double t = fma(u, 4.0, RND52);
  sincos_quarters(fma(t - RND52, -0.25, u), __double2loint(t), s, c);
}
// sin and cos of x radians: the turns x / 2 pi less the nearest quarter by multiply-adds with both parts of
// 1 / 2 pi, so that the reduced angle has no error but its own rounding.  20 FP64 operations.
__device__ __forceinline__ void sincos_radians(double x, double* s, double* c) {
  const double hi = 0.15915494309189535, lo = -9.839338337591243e-18;  // 1 / 2 pi
  const double t = fma(x, 4.0 * hi, RND52);
  sincos_quarters(fma(x, lo, fma(x, hi, -0.25 * (t - RND52))), __double2loint(t), s, c);
}

// sin of 2 pi r for |r| <= 1/4 (a polynomial of degree 8 in r^2 times r, a Chebyshev fit; within
// 2.6e-16 of the value, relative near 0), and of 2 pi u for any |u| < 2^50, reduced exactly by the
// nearest half turn.  10 and 13 FP64 operations.
// The coefficients are read from constant memory: an FP64 multiply-add takes an operand from there,
// while 64-bit literals are moved into registers first, a fifth of the grain kernel's instructions.
static __constant__ double SIN_TURN[9] = {6.283185307179586,  -41.341702240399755, 81.60524927607344,
                                          -76.70585975280203, 42.058693924097824,  -15.094641633983702,
                                          3.8199273419380186, -0.7177266693115234, 0.100869140625};
__device__ __forceinline__ double sin_quarter_turn(double r) {
  const double z = r * r;
  double p = SIN_TURN[8];
#pragma unroll
  for (int i = 7; i >= 0; --i) p = fma(p, z, SIN_TURN[i]);
  return p * r;
}
__device__ __forceinline__ double sin_turns(double u) {
  const double t = fma(u, 2.0, RND52);
  const double s = sin_quarter_turn(fma(t - RND52, -0.5, u));
  return __hiloint2double(__double2hiint(s) ^ (__double2loint(t) << 31), __double2loint(s));
}

}  // namespace hgx
