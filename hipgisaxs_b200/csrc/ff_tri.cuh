// Shared by the triangle form-factor kernels (ff_tri.cu, ff_tri_mma.cu): tile layout, rotation,
// phase and output helpers.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "hgx_internal.cuh"

namespace hgx {

constexpr int TILE = TRI_TILE;              // triangles per shared-memory tile (512)
constexpr int TILE_FLOATS = TILE * 6;       // float4 A[TILE] (dx,nx,dy,ny) + float2 B[TILE] (dz,nz)
constexpr uint32_t TILE_BYTES = TILE_FLOATS * 4;
constexpr double TWO_PI = 6.283185307179586476925286766559;
constexpr double INV_TWO_PI = 0.15915494309189533576888376337251;
constexpr float TWO_PI_F = 6.28318530717958648f;
constexpr float INV_TWO_PI_F = 0.159154943091895336f;
// In-plane phases of a tile with |q_par| * (largest offset) above 8 pi radians get the
// explicit reduction to [-1/2, 1/2] turn before the SFU; below it they go straight in (the SFU
// reduces its argument itself; its error grows with |x| by the rounding of x / 2 pi, about
// 2^-24 |x|, 1.5e-6 rad at 8 pi).
constexpr float WIDE_PHASE2 = 631.65468f;   // (8 pi)^2

struct Rot9 {
  double r[9];
};

// |R (qx, qy, qz)|^2 with complex qz, as RotMatrix_t::rotate + cuCnorm3 evaluate it.
__device__ __forceinline__ double rotated_q2(const Rot9& R, double qx, double qy, double2 qz) {
  double q2 = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double re = R.r[3 * j] * qx + R.r[3 * j + 1] * qy + R.r[3 * j + 2] * qz.x;
    double im = R.r[3 * j + 2] * qz.y;
    q2 += re * re + im * im;
  }
  return q2;
}

template <typename OUT>
__device__ __forceinline__ void store_ff(OUT* out, long idx, double re, double im);
template <>
__device__ __forceinline__ void store_ff<float2>(float2* out, long idx, double re, double im) {
  out[idx] = make_float2((float)re, (float)im);
}
template <>
__device__ __forceinline__ void store_ff<double2>(double2* out, long idx, double re, double im) {
  out[idx] = make_double2(re, im);
}

// The anchor phasor e^{2 pi i u} of an FP64 phase u in turns, reduced exactly in FP64.
__device__ __forceinline__ float2 anchor_phasor(double u) {
  u -= rint(u);
  float s, c;
  sincospif((float)(2.0 * u), &s, &c);
  return make_float2(c, s);
}

// (re, im) <- (re, im) * (c + i s)
__device__ __forceinline__ void rotate_pair(float& re, float& im, float2 a) {
  const float r = re * a.x - im * a.y;
  im = re * a.y + im * a.x;
  re = r;
}

// Rounds x to the nearest integer (ties to even) with two FP32 adds — valid for
// |x| < 2^22 — so the reduction stays on the FMA pipe instead of the conversion unit.
__device__ __forceinline__ float round_nearest(float x) {
  const float magic = 12582912.0f;  // 1.5 * 2^23
  return (x + magic) - magic;
}

__device__ __forceinline__ void two_sum_fold(float& sum, float& part, float& comp) {
  float s = sum + part;
  float bp = s - sum;
  float err = (sum - (s - bp)) + (part - bp);
  sum = s;
  comp += err;
  part = 0.f;
}

// Row factor of one (row, triangle) for a real block pair (qz, -qz), cz in turns (FP64):
// Z = e^{i 2pi qz cz} = (x, y), D = qz n~z; returns (x, y, D*y, D*x).
__device__ __forceinline__ float4 paired_factor(double q, double cz, float nz) {
  double u = q * cz;
  u -= rint(u);
  float s, c;
  sincospif((float)(2.0 * u), &s, &c);
  float D = (float)(q * (double)nz);
  return make_float4(c, s, D * s, D * c);
}

// Row factor for a general complex block, cz in turns: Z = e^{i 2pi qz cz}, D = qz n~z;
// returns (Z, D Z).
__device__ __forceinline__ float4 complex_factor(double2 q, double cz, float nz) {
  double u = q.x * cz;
  u -= rint(u);
  double amp = exp(-TWO_PI * q.y * cz);
  double s, c;
  sincospi(2.0 * u, &s, &c);
  double zr = amp * c, zi = amp * s;
  double dr = q.x * (double)nz, di = q.y * (double)nz;
  return make_float4((float)zr, (float)zi, (float)(dr * zr - di * zi), (float)(dr * zi + di * zr));
}

}  // namespace hgx
