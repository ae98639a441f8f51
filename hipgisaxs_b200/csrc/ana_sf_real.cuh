// Bodies of the fused grain kernel (hig_sim.cu) for real qz (grids whose DWBA blocks are real: a
// vacuum particle layer), T = double (FP64) or float (FP32C): the cylinder, sphere and box form
// factors and the lattice structure factor of ana_sf.cuh's formulas in real arithmetic.  FP32C
// forms and reduces every phase in FP64 and takes the transcendental of the reduced argument and
// the sums in FP32.
//
// Lattice structure factor: for a real angle the reference's principal-branch complex powers
//   pow(e, (1 - N)/2) (1 - pow(e, N)) / (1 - e),  e = e^{i theta}  (src/sf/sf.cpp:164-246)
// are sin(N theta_r / 2) / sin(theta_r / 2) with theta_r the principal angle of e.  On the b axis
// the reference's numerator is 1 - e^{i N theta} of the unreduced theta = theta_r + 2 pi k: the same
// for a whole N, sin(N theta / 2) / sin(theta_r / 2) e^{i pi k N} for another (dirichlet_b_real,
// b_phase_real).  N is returned at theta_r = 0, where the reference's guard takes N.  Two sines
// instead of five complex exponentials, four powers and three divisions; angles in turns, so that
// their reduction is exact.
//
// Form factors: sinc(x) e^{ix} terms as one sincos; the cylinder's evenly stepped heights in
// closed form (ana_sf_f32.cuh) where the samples step to rounding (FP64: prog == 2).
#pragma once

#include "ana_sf.cuh"
#include "ana_sf_f32.cuh"
#include "turns.cuh"

namespace hgx {

constexpr double INV_2PI_R = 0.15915494309189533576888376337251;

template <typename T>
struct cx {
  T x, y;
};
template <typename T>
__device__ __forceinline__ cx<T> operator+(cx<T> a, cx<T> b) { return cx<T>{a.x + b.x, a.y + b.y}; }
template <typename T>
__device__ __forceinline__ cx<T> operator*(cx<T> a, cx<T> b) {
  return cx<T>{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename T>
__device__ __forceinline__ cx<T> operator*(T s, cx<T> a) { return cx<T>{s * a.x, s * a.y}; }

// e^{2 pi i u}, e^{i ph}
template <typename T>
__device__ __forceinline__ cx<T> expi_turns_real(double u);
template <>
__device__ __forceinline__ cx<double> expi_turns_real<double>(double u) {
  double s, c;
  sincos_turns(u, &s, &c);
  return cx<double>{c, s};
}
template <>
__device__ __forceinline__ cx<float> expi_turns_real<float>(double u) {
  const cf e = expi_turns(u);
  return cx<float>{e.x, e.y};
}
template <typename T>
__device__ __forceinline__ cx<T> expi_real(double ph);
template <>
__device__ __forceinline__ cx<double> expi_real<double>(double ph) {
  double s, c;
  sincos_radians(ph, &s, &c);
  return cx<double>{c, s};
}
template <>
__device__ __forceinline__ cx<float> expi_real<float>(double ph) { return expi_turns_real<float>(ph * INV_2PI_R); }

// a / b without the branches of the IEEE division, for 1e-37 < |b| < 1e37 (sines and phases here): b's
// reciprocal from the approximate one (FP64: two Newton steps), the quotient corrected by its remainder; rounded
// as the IEEE division is but for rare ties.  CORRECT = false: without the correction, within two ulp.
template <bool CORRECT = true>
__device__ __forceinline__ double quotient(double a, double b) {
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"((float)b));
  double y = (double)y0;
  y = fma(y, fma(-b, y, 1.0), y);
  y = fma(y, fma(-b, y, 1.0), y);
  const double q = a * y;
  return CORRECT ? fma(fma(-b, q, a), y, q) : q;
}
template <bool CORRECT = true>
__device__ __forceinline__ float quotient(float a, float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  const float q = a * y;
  return CORRECT ? fmaf(fmaf(-b, q, a), y, q) : q;
}
// The same of a lattice factor: corrected in FP32C, whose sines are as good; in FP64 the rounding of the
// angles, some 1e-14 of the factor, leaves nothing to correct (7.0e-15 norm-wise either way).
__device__ __forceinline__ double lattice_quotient(double a, double b) { return quotient<false>(a, b); }
__device__ __forceinline__ float lattice_quotient(float a, float b) { return quotient(a, b); }

// sin(x) / x (hig::sinc for a real x) given sin x
__device__ __forceinline__ double sinc_real(double x, double sinx) {
  return fabs(x) > 1.0e-14 ? quotient(sinx, x) : 1.0;
}
__device__ __forceinline__ float sinc_real(double x, float sinx) { return sinc_from(x, sinx); }

// A lattice factor as num / den at the angle of `u` turns; N itself within 1e-13 turn of a whole
// one, where the ratio is N to rounding (the products of two denominators then stay in range).
// FULL: the numerator takes the unreduced angle, and N is the value at a whole number of turns only
// (elsewhere near one the ratio is far from N unless that number is 0).
template <typename T>
struct Ratio {
  T num, den;
};
template <typename T>
__device__ __forceinline__ Ratio<T> dirichlet_real(double u, double N, bool full = false);
template <>
__device__ __forceinline__ Ratio<double> dirichlet_real<double>(double u, double N, bool full) {
  const double t = u - round_fp64(u), h = 0.5 * t;
  const double n = sin_turns(N * (full ? 0.5 * u : h)), d = sin_quarter_turn(h);
  const bool zero = full ? t == 0.0 : fabs(t) < 1e-13;
  return Ratio<double>{zero ? N : n, zero ? 1.0 : d};
}
template <>
__device__ __forceinline__ Ratio<float> dirichlet_real<float>(double u, double N, bool full) {
  const double t = u - round_fp64(u);
  const double v = N * (full ? u : t), kv = v + RND52;  // nearest integer in the low mantissa bits
  const float n = sin_half_turn((float)(v - (kv - RND52))), d = sin_half_turn((float)t);
  const float sn = __int_as_float(__float_as_int(n) ^ (__double2loint(kv) << 31));
  const bool zero = full ? t == 0.0 : fabs(t) < 1e-13;
  return Ratio<float>{zero ? (float)N : sn, zero ? 1.0f : d};
}

// The b axis' factor, and its phase where N is not whole.
template <typename T>
__device__ __forceinline__ Ratio<T> dirichlet_b_real(double u, double N) {
  return dirichlet_real<T>(u, N, N != round_fp64(N));
}
template <typename T>
__device__ __forceinline__ cx<T> b_phase_real(double u, double N) {
  const double k = round_fp64(u);
  return expi_turns_real<T>(u == k ? 0.0 : 0.5 * k * N);
}

// The cylinder's radial sum over its samples (unweighted), ff_ana_cylinder.cpp:34-42,100-117.
// Out of line, as the other sums: one copy of the Bessel function for the kernel.
template <typename T>
static __device__ __noinline__ T cyl_radial_real(const Dist& X, double qpar) {
  T fr = 0;
  for (int i = 0; i < X.n; ++i) {
    const double r = X.v[i], x = qpar * r;
    if (x * x > CUTINY_REF) {
      if (sizeof(T) == 8) fr += (T)(quotient(j1(x), x) * (2. * PI_REF * r * r));
      else fr += (T)((float)(2. * PI_REF * r * r) * (j1f((float)x) / (float)x));
    }
  }
  return fr;
}

// sum_j h_j sinc(qz h_j/2) e^{i qz h_j/2}, each term (e^{i qz h_j} - 1) / (i qz)
template <typename T>
static __device__ __noinline__ cx<T> cyl_axial_real(const Dist& Z, double qz) {
  if (sizeof(T) == 4) {
    const cf v = cyl_height_sum_f32(Z, qz);
    return cx<T>{(T)v.x, (T)v.y};
  }
  const int n = Z.n;
  if (Z.prog == 2 && fabs(qz) * fmax(fabs(Z.v[0]), fabs(Z.v[n - 1])) >= 0.5) {
    const double u = qz * ((Z.v[n - 1] - Z.v[0]) / (n - 1)) * INV_2PI_R, k = round_fp64(u);
    const Ratio<double> d = dirichlet_real<double>(u, (double)n);
    // sin(n pi u) / sin(pi u) at the unreduced u: (-1)^(k (n - 1)) times the principal one
    const bool flip = ((n - 1) & 1) && 0.5 * k != round_fp64(0.5 * k);
    const double D = flip ? -d.num / d.den : d.num / d.den;
    const cx<double> e = expi_real<double>(qz * 0.5 * (Z.v[0] + Z.v[n - 1]));
    const double iq = 1.0 / qz;
    return cx<T>{(T)(e.y * D * iq), (T)(((double)n - e.x * D) * iq)};
  }
  cx<T> gh{0, 0};
  for (int i = 0; i < n; ++i) {
    const double h = Z.v[i], x = qz * 0.5 * h;
    const cx<T> e = expi_real<T>(x);
    gh = gh + (sinc_real(x, e.y) * (T)h) * e;
  }
  return gh;
}

// The box's sum over one in-plane axis, sum_j w_j x_j sinc(q x_j / 2) (ff_ana_box.cpp:35-42,96-125),
// and its height sum with e^{i q z_j / 2}.
template <typename T>
static __device__ __noinline__ T box_side_real(const Dist& X, double q) {
  T s = 0;
  for (int i = 0; i < X.n; ++i) {
    const double x = q * 0.5 * X.v[i];
    s += sinc_real(x, expi_real<T>(x).y) * (T)(X.v[i] * X.w[i]);
  }
  return s;
}
template <typename T>
static __device__ __noinline__ cx<T> box_axial_real(const Dist& Z, double qz) {
  cx<T> s{0, 0};
  for (int i = 0; i < Z.n; ++i) {
    const double x = qz * 0.5 * Z.v[i];
    const cx<T> e = expi_real<T>(x);
    s = s + (sinc_real(x, e.y) * (T)(Z.v[i] * Z.w[i])) * e;
  }
  return s;
}

// (sin x - x cos x) / x^3, below 1/2 its series (the next term is below 3e-18)
__device__ __forceinline__ double sphere_kernel(double x, double) {
  if (x < 0.5) {
    const double z = x * x;
    return 1. / 3. - z * (1. / 30. - z * (1. / 840. - z * (1. / 45360. - z * (1. / 3991680. -
                     z * (1. / 518918400. - z * (1. / 93405312000.))))));
  }
  const cx<double> e = expi_real<double>(x);
  return (e.y - x * e.x) / (x * x * x);
}
__device__ __forceinline__ float sphere_kernel(double x, float) { return sphere_kernel_f(x); }

// ff_ana_sphere.cpp:33-45,95-107 (weighted)
template <typename T>
static __device__ __noinline__ cx<T> sphere_real(const Dist& X, double m0, double m1, double m2) {
  const double q = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
  cx<T> acc{0, 0};
  if (q < 2.2250738585072014e-308) return acc;
  for (int i = 0; i < X.n; ++i) {
    const double R = X.v[i];
    acc = acc + (sphere_kernel(q * R, T()) * (T)(4 * PI_REF * R * R * R * X.w[i])) * expi_real<T>(m2 * R);
  }
  return acc;
}

// The parts of a cylinder or box form factor that depend on the rotated in-plane q and on the
// rotated qz: ff = in-plane x axial.
template <typename T, int SHAPE>
__device__ __forceinline__ T ff_inplane_real(const AnaShape& a, double m0, double m1) {
  if (SHAPE == SH_CYLINDER) return cyl_radial_real<T>(a.d[0], sqrt(m0 * m0 + m1 * m1));
  return box_side_real<T>(a.d[0], m0) * box_side_real<T>(a.d[1], m1);
}
template <typename T, int SHAPE>
__device__ __forceinline__ cx<T> ff_axial_real(const AnaShape& a, double m2) {
  if (SHAPE == SH_CYLINDER) return cyl_axial_real<T>(a.d[2], m2);
  return box_axial_real<T>(a.d[2], m2);
}

}  // namespace hgx
