// FP64 bodies of the fused grain kernel (hig_sim.cu) for real qz (grids whose DWBA blocks are
// real: a vacuum particle layer): the cylinder, sphere and box form factors and the lattice
// structure factor of ana_sf.cuh's formulas, in real arithmetic.
//
// Lattice structure factor: for a real angle the reference's principal-branch complex powers
//   pow(e, (1 - N)/2) (1 - pow(e, N)) / (1 - e),  e = e^{i theta}  (src/sf/sf.cpp:164-246)
// are sin(N theta_r / 2) / sin(theta_r / 2) with theta_r the principal angle of e; on the b axis
// the numerator takes the unreduced theta, which for a non-integer N adds the phase
// e^{i pi k (N - 1)}, theta = theta_r + 2 pi k.  N is returned at theta_r = 0, where the reference's
// guard takes N.  Two sines instead of five complex exponentials, four powers and three divisions;
// phases in turns, so that their reduction is exact.
//
// Form factors: q-space sinc(x) e^{ix} terms as one sincos; the cylinder's evenly stepped heights
// in closed form (ana_sf_f32.cuh) where the samples step to rounding (prog == 2).
#pragma once

#include "ana_sf.cuh"
#include "turns.cuh"

namespace hgx {

constexpr double INV_2PI_R = 0.15915494309189533576888376337251;

__device__ __forceinline__ zd expi_real(double ph) {  // e^{i ph}
  double s, c;
  sincos_turns(ph * INV_2PI_R, &s, &c);
  return zd(c, s);
}

// sin(x) / x (hig::sinc for a real x) given sin x
__device__ __forceinline__ double sinc_real(double x, double sinx) {
  return fabs(x) > 1.0e-14 ? sinx / x : 1.0;
}

// A lattice factor as num / den at the angle of `u` turns.
struct Ratio {
  double num, den;
};
__device__ __forceinline__ Ratio dirichlet_real(double u, double N) {
  const double t = u - round_fp64(u);
  if (t == 0.0 || N == 1.0) return Ratio{N, 1.0};
  const double h = 0.5 * t;
  return Ratio{sin_turns(N * h), sin_quarter_turn(h)};
}
// The phase e^{i pi k (N - 1)} of the b axis (1 for an integer N).
__device__ __forceinline__ zd dirichlet_b_phase(double u, double N) {
  if (N == round_fp64(N)) return zd(1.0, 0.0);
  double s, c;
  sincos_turns(0.5 * round_fp64(u) * (N - 1.0), &s, &c);
  return zd(c, s);
}

// The cylinder's radial sum over its samples (unweighted), ff_ana_cylinder.cpp:34-42,100-117.
// Out of line: one copy of the Bessel function for the kernel.
static __device__ __noinline__ double cyl_radial_real(const Dist& X, double qpar) {
  double fr = 0.0;
  for (int i = 0; i < X.n; ++i) {
    const double r = X.v[i], x = qpar * r;
    if (x * x > CUTINY_REF) fr += j1(x) / x * (2. * PI_REF * r * r);
  }
  return fr;
}

// sum_j h_j sinc(qz h_j/2) e^{i qz h_j/2}, each term (e^{i qz h_j} - 1) / (i qz)
static __device__ __noinline__ zd cyl_axial_real(const Dist& Z, double qz) {
  const int n = Z.n;
  if (Z.prog == 2 && fabs(qz) * fmax(fabs(Z.v[0]), fabs(Z.v[n - 1])) >= 0.5) {
    const Ratio d = dirichlet_real(qz * ((Z.v[n - 1] - Z.v[0]) / (n - 1)) * INV_2PI_R, (double)n);
    // the closed form's sign over whole turns of a single step, (-1)^(k (n-1)), is not dropped
    const double k = round_fp64(qz * ((Z.v[n - 1] - Z.v[0]) / (n - 1)) * INV_2PI_R);
    const bool flip = ((n - 1) & 1) && 0.5 * k != round_fp64(0.5 * k);
    const double D = flip ? -d.num / d.den : d.num / d.den;
    const zd e = expi_real(qz * 0.5 * (Z.v[0] + Z.v[n - 1]));
    const double iq = 1.0 / qz;
    return zd(e.y * D * iq, ((double)n - e.x * D) * iq);
  }
  zd gh(0, 0);
  for (int i = 0; i < n; ++i) {
    const double h = Z.v[i], x = qz * 0.5 * h;
    const zd e = expi_real(x);
    gh += e * (sinc_real(x, e.y) * h);
  }
  return gh;
}

// The box's sum over one in-plane axis, sum_j w_j x_j sinc(q x_j / 2) (ff_ana_box.cpp:35-42,96-125),
// and its height sum with e^{i q z_j / 2}.
static __device__ __noinline__ double box_side_real(const Dist& X, double q) {
  double s = 0.0;
  for (int i = 0; i < X.n; ++i) {
    const double x = q * 0.5 * X.v[i];
    s += sinc_real(x, sin_turns(x * INV_2PI_R)) * (X.v[i] * X.w[i]);
  }
  return s;
}
static __device__ __noinline__ zd box_axial_real(const Dist& Z, double qz) {
  zd s(0, 0);
  for (int i = 0; i < Z.n; ++i) {
    const double x = qz * 0.5 * Z.v[i];
    const zd e = expi_real(x);
    s += e * (sinc_real(x, e.y) * (Z.v[i] * Z.w[i]));
  }
  return s;
}

// ff_ana_sphere.cpp:33-45,95-107 (weighted)
static __device__ __noinline__ zd sphere_real(const Dist& X, double m0, double m1, double m2) {
  const double q = sqrt(m0 * m0 + m1 * m1 + m2 * m2);
  zd acc(0, 0);
  if (q < 2.2250738585072014e-308) return acc;
  for (int i = 0; i < X.n; ++i) {
    const double R = X.v[i], x = q * R;
    const zd e = expi_real(x);
    const double c0 = (e.y - x * e.x) / (x * x * x);
    acc += expi_real(m2 * R) * (c0 * (4 * PI_REF * R * R * R) * X.w[i]);
  }
  return acc;
}

// The parts of a cylinder or box form factor that depend on the rotated in-plane q and on the
// rotated qz: ff = in-plane x axial.
template <int SHAPE>
__device__ __forceinline__ double ff_inplane_real(const AnaShape& a, double m0, double m1) {
  if (SHAPE == SH_CYLINDER) return cyl_radial_real(a.d[0], sqrt(m0 * m0 + m1 * m1));
  return box_side_real(a.d[0], m0) * box_side_real(a.d[1], m1);
}
template <int SHAPE>
__device__ __forceinline__ zd ff_axial_real(const AnaShape& a, double m2) {
  if (SHAPE == SH_CYLINDER) return cyl_axial_real(a.d[2], m2);
  return box_axial_real(a.d[2], m2);
}

}  // namespace hgx
