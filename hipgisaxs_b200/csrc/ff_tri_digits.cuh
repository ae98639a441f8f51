// Fixed-point digits for tcgen05.mma kind::i8, shared by the triangle form factor (ff_tri_mma.cu) and
// its adjoint (mesh_adjoint_mma.cu): phasors as three signed 8-bit digits, value = d0 2^16 + d1 2^8 + d2, the
// other factor as four.
#pragma once

#include "ff_tri.cuh"

namespace hgx {

constexpr int MMA_K = 32;                     // triangles per product
constexpr float A_SCALE = 4161344.0f;         // |c| <= 1 -> below 2^22 - 0x8080, so the sum below stays under 2^23
constexpr float A_MAGIC = 12615808.0f;        // 2^23 + 2^22 + 0x8080: low mantissa bits = a + 2^22 + 0x8080
constexpr double B_SCALE = 8355000.0 * 256.0; // the largest of the other factor (four signed digits reach 0x7f7f7f7f)
// One unit (2^16 products) of the combined sum.  The sums are taken in units of 2^36 of these and the scales
// times 2^36 (about half the largest factor), so that neither leaves the range of FP32 where the factors do not.
constexpr float S36 = 1.0f / 68719476736.0f;
constexpr double V_UNIT = 65536.0 / (4161344.0 * B_SCALE) * 68719476736.0;

constexpr int A_COLS = 6 * MMA_K / 4;          // TMEM columns of a warpgroup's digits (2 x 3 planes of 8)

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { return __byte_perm(a, b, sel); }

// The digit planes of four integers b_i = w_i - 0x80808080, |b_i| <= 0x7f7f7f7f, one byte each.
__device__ __forceinline__ void signed_digits(const uint32_t (&w)[4], uint32_t (&dig)[4]) {
  const uint32_t p01 = prmt(w[0], w[1], 0x5140), p23 = prmt(w[2], w[3], 0x5140);
  const uint32_t h01 = prmt(w[0], w[1], 0x7362), h23 = prmt(w[2], w[3], 0x7362);
  dig[0] = prmt(h01, h23, 0x7632) ^ 0x80808080u;
  dig[1] = prmt(h01, h23, 0x5410) ^ 0x80808080u;
  dig[2] = prmt(p01, p23, 0x7632) ^ 0x80808080u;
  dig[3] = prmt(p01, p23, 0x5410) ^ 0x80808080u;
}

// The offset of 64 of the phasors' top digits adds 2^22 sum(b) to a column's sum: in units of 2^32, and the rest
// in the combined sum's.
__device__ __forceinline__ uint32_t offset_units(long long sum) { return (uint32_t)(sum >> 10); }
__device__ __forceinline__ float offset_rest(long long sum) { return (float)((int)(sum & 1023) << 6) * S36; }
// A column's combined sum less that offset, from its four accumulators s_i (weights 2^24, 2^16, 2^8, 1 units):
// the low two's part, and the whole.
__device__ __forceinline__ float low_sum(uint32_t s2, uint32_t s3, float rest) {
  return fmaf((float)(int)s2, 256.f * S36, fmaf((float)(int)s3, S36, -rest));
}
__device__ __forceinline__ float combined_sum(uint32_t s0, uint32_t s1, uint32_t units, float low) {
  return fmaf((float)(int)(s0 * 256u + s1 - units), 65536.f * S36, low);
}

// The digits of the phasors e^{i q.d} of this thread's q with 16 offsets d (or of its offset with
// 16 q; xy: (x0, x1, y0, y1) per pair): w[4 p + g] holds plane p (0-2 cos, 3-5 sin) of numbers 4 g
// .. 4 g + 3.  The top digit carries an offset of 64 (0 .. 127).  WIDE: the phases get the explicit reduction.
template <bool WIDE>
__device__ __forceinline__ void phasor_digits(const float4* __restrict__ xy, float qx, float qy, uint32_t (&w)[24]) {
  const float2 q0 = make_float2(qx, qx), q1 = make_float2(qy, qy);
  const float2 sc = make_float2(A_SCALE, A_SCALE), mg = make_float2(A_MAGIC, A_MAGIC);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t x[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 v = xy[2 * g + h];
      float2 tp = __ffma2_rn(q0, make_float2(v.x, v.y), __fmul2_rn(q1, make_float2(v.z, v.w)));
      if (WIDE) {
        float t0 = tp.x * INV_TWO_PI_F, t1 = tp.y * INV_TWO_PI_F;
        tp.x = (t0 - round_nearest(t0)) * TWO_PI_F;
        tp.y = (t1 - round_nearest(t1)) * TWO_PI_F;
      }
      float s0, c0, s1, c1;
      __sincosf(tp.x, &s0, &c0);
      __sincosf(tp.y, &s1, &c1);
      const float2 fc = __ffma2_rn(make_float2(c0, c1), sc, mg), fs = __ffma2_rn(make_float2(s0, s1), sc, mg);
      x[0][2 * h] = __float_as_uint(fc.x);
      x[0][2 * h + 1] = __float_as_uint(fc.y);
      x[1][2 * h] = __float_as_uint(fs.x);
      x[1][2 * h + 1] = __float_as_uint(fs.y);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t p01 = prmt(x[k][0], x[k][1], 0x5140), p23 = prmt(x[k][2], x[k][3], 0x5140);
      const uint32_t h01 = prmt(x[k][0], x[k][1], 0x0062), h23 = prmt(x[k][2], x[k][3], 0x0062);
      w[12 * k + g] = prmt(h01, h23, 0x5410);                       // top digit + 64, in 0 .. 127
      w[12 * k + 4 + g] = prmt(p01, p23, 0x7632) ^ 0x80808080u;
      w[12 * k + 8 + g] = prmt(p01, p23, 0x5410) ^ 0x80808080u;
    }
  }
}

// One warpgroup's barrier.
__device__ __forceinline__ void wg_sync(int wg) { asm volatile("bar.sync %0, 128;" ::"r"(wg + 1) : "memory"); }

}  // namespace hgx
