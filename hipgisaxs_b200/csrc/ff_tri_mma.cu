// FP32C triangle form factor on row grids, its sums on the tensor cores.
//
// For one detector row the sums over a tile's triangles are a matrix product: with the in-plane
// phasor e^{i(qx dx + qy dy)} = c + i s of each (pixel, triangle) and the row factor
// Z = e^{i qz c'z} of each (row, triangle),
//   sum_t (q.n~) e^{iq.d} Z = qx sum (c+is) n~x Z + qy sum (c+is) n~y Z + qz sum (c+is) n~z Z,
// so the tile needs sum_t c_t b_tj and sum_t s_t b_tj with the six real columns
// b = (n~x, n~y, n~z) x (Re Z, Im Z) per block pair (qz, -qz) or per complex block.
//
// Both factors become fixed-point integers cut into signed 8-bit digits: |c|, |s| <= 1 with step
// 1 / 4161344 (about 2^-22) into three, the row factors relative to the tile's largest |n~| (step
// 2^-31, so that those of triangles of 2^-7 of the largest still have their 24 bits) into four.  The
// products of digits with i + j <= 3 accumulate exactly in 32-bit integers (tcgen05.mma kind::i8, A =
// the phasors in TMEM, B = the row factors in shared memory, accumulators in TMEM):
//   A0 x [B0 B1 B2 B3], A1 x [B0 B1 B2], A2 x [B0 B1], the slices offset so that equal i + j add up.
// What is left out is below 2^-29 of a term, and the accumulation itself has no rounding error.
// Norm-wise error over the FP32 row kernel's: 0.6 to 0.7 on closed meshes of even and of uneven
// triangles, 0.3 to 0.5 on complex blocks (with three digits, step 2^-23: 0.7 on even ones, up to 3 on uneven
// ones, and 5 to 11 on complex blocks), 1.2 where pairs of opposite faces a thousandth of a nm apart cancel
// to 1e-4, where the phasors' step shows.
//
// A CTA (one per SM) owns 128 columns of one detector row, the 128 TMEM lanes, and a range of
// tiles.  Five warpgroups take its chunks of 32 triangles in turn: each
// thread makes its pixel's digits and stores them to its warpgroup's part of TMEM; two more warps
// issue the products with cos and with sin.  On real blocks the accumulators alternate between
// two column ranges, so that a tile's sums are read back, scaled, rotated by the tile's FP64
// anchor phasor and added to FP64 sums (in shared memory) by one warpgroup while the others go
// on with the next tile.
//
// What bounds it: the digits.  Per (pixel, triangle) two SFU operations and about 14 issued
// instructions (PRMT 3.6, FFMA2 1.5, LOP3 1.3, FMUL 1.2): SFU 76%, issue 66%; the products take
// 150 of the 690 cycles of a chunk.  2048 x 2048 x 50,000: 128 ms with 20 digit warps of 80
// registers (with three digits of the row factors 126, and then 24 warps of 72: 129, 16 of 96: 147, three
// warpgroups of 168 registers, each with its own pixels: 148), against 190 ms for the FP32 row kernel, whose 16
// FFMA per (pixel, triangle) of accumulation these products replace.  Taking a quarter of the sines off the SFU by polynomials on the
// FMA pipe left the time unchanged.
//
// The row factors of a slab of rows are made once per (row, triangle) by ff_row_factor_kernel,
// in the layout the tensor core reads, and fetched by bulk copies; 128-column items of a row
// share them through L2.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "ff_tri_digits.cuh"
#include "ff_tri_rows.cuh"
#include "ptx.cuh"
#include "tc05.cuh"

namespace hgx {

constexpr int MMA_CHUNKS = TILE / MMA_K;      // products per full tile

// Layout of one kind of grid: U row-factor units (block pairs or complex blocks) of six columns.
template <int U>
struct MmaShape {
  static constexpr int NP = U == 4 ? 32 : 16;           // columns per digit slice (6 U, padded)
  static constexpr int SBO = 128;
  static constexpr int LBO = 4 * NP / 8 * 128;
  static constexpr int CHUNK_BYTES = 2 * LBO;           // row factors of 32 triangles
  static constexpr int TILE_B_BYTES = MMA_CHUNKS * CHUNK_BYTES;
  static constexpr int XY_BYTES = MMA_XY * 4;
  static constexpr int REC = (13 * U + 3) / 4 * 4;      // words per (row, tile) record
  static constexpr int STAGE = TILE_B_BYTES + XY_BYTES + REC * 4;  // one tile in shared memory
  static constexpr int NST = U == 4 ? 2 : 4;            // tiles in shared memory
  static constexpr int D_COLS = 4 * NP;                 // accumulator columns of cos, then of sin
  static constexpr int DBUF = U == 4 ? 1 : 2;           // accumulator ranges
  static constexpr int SUB = 5;                         // warpgroups making digits
  static constexpr int THREADS = SUB * 128 + 64;        // and two warps that issue the products
  static constexpr int NACC = U == 1 ? 2 : 8;           // sums per pixel
  static constexpr int SUM_BYTES = SUB * NACC * 128 * 8;  // FP64 sums of each warpgroup
  static constexpr int SMEM = NST * STAGE + SUM_BYTES + 128 * 8 * 8;  // and the sums next to q = 0
};

// ------------------------------------------------------------- row factors ----
struct FactorArgs {
  const float* tiles;
  const double4* anchors;
  const float4* info;      // per tile: largest |n~|, smallest and largest dz
  const double2* rowqz;    // nrow x NK
  int ntiles, row0, nrows; // slab rows
  unsigned char* b;        // [slab row][tile] TILE_B_BYTES
  uint32_t* rec;           // [slab row][tile] REC words: 6 U offsets, U scales, 6 U offsets' rests
};

constexpr int FACTOR_THREADS = TILE / 4;

// One CTA per tile and group of rows, four triangles per thread (one 32-bit word of each digit
// plane).  The digits are biased by 0x80 (the bytes of b + 0x80808080) and flipped back to signed
// bytes; the tile's image is put together in shared memory and written out in 16-byte words.
// About 200 instructions per (row, triangle), 1% of the products' time at 2048 columns.
template <int U, bool PAIRED>
__global__ void __launch_bounds__(FACTOR_THREADS) ff_row_factor_kernel(FactorArgs a) {
  using S = MmaShape<U>;
  constexpr int NK = PAIRED ? 4 : U;
  extern __shared__ __align__(16) unsigned char s_img[];
  __shared__ long long s_sum[FACTOR_THREADS / 32][6 * U];
  const int tile = blockIdx.x, t = threadIdx.x;
  const double4 anc = a.anchors[tile];
  const float4 info = a.info[tile];
  const double sc = info.x > 0.f ? B_SCALE / (double)info.x : 0.0;
  const double cz0 = anc.z * INV_TWO_PI;
  const double zlo = cz0 + (double)info.y * INV_TWO_PI, zhi = cz0 + (double)info.z * INV_TWO_PI;
  const float4* A = reinterpret_cast<const float4*>(a.tiles + (size_t)tile * TILE_FLOATS);
  const float2* B = reinterpret_cast<const float2*>(a.tiles + (size_t)tile * TILE_FLOATS + 4 * TILE);
  float n[4][3];
  double cz[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = A[4 * t + i];
    const float2 z = B[4 * t + i];
    n[i][0] = (float)(v.y * sc);
    n[i][1] = (float)(v.w * sc);
    n[i][2] = (float)(z.y * sc);
    cz[i] = cz0 + (double)z.x * INV_TWO_PI;
  }
  for (int i = t; i < S::TILE_B_BYTES / 16; i += FACTOR_THREADS)
    reinterpret_cast<uint4*>(s_img)[i] = make_uint4(0, 0, 0, 0);  // padding columns stay zero
  __syncthreads();
  // byte offset of triangles 4t .. 4t + 3 in column 0
  const int base = (t >> 3) * S::CHUNK_BYTES + ((t >> 2) & 1) * S::LBO + (t & 3) * 4;
  for (int r = blockIdx.y; r < a.nrows; r += gridDim.y) {
    const size_t cell = (size_t)r * a.ntiles + tile;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 q = a.rowqz[(long)(a.row0 + r) * NK + (PAIRED ? 2 * u : u)];
      float re[4], im[4];
      double top = 1.0;  // the block's largest amplitude in the tile
      if (PAIRED) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          double w = q.x * cz[i];
          w -= rint(w);
          sincospif((float)(2.0 * w), &im[i], &re[i]);
        }
      } else {
        const double ze = q.y > 0.0 ? zlo : zhi;  // where e^{-Im(qz) z} is largest
        top = exp(-TWO_PI * q.y * ze);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          double w = q.x * cz[i];
          w -= rint(w);
          double s, c;
          sincospi(2.0 * w, &s, &c);
          const double amp = q.y == 0.0 ? 1.0 : exp(-TWO_PI * q.y * (cz[i] - ze));
          re[i] = (float)(amp * c);
          im[i] = (float)(amp * s);
        }
      }
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        uint32_t w[4];
        int hi = 0, lo = 0;  // of the sum of b, so that a warp's fits
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b = __float2int_rn(n[i][j % 3] * (j < 3 ? re[i] : im[i]));
          hi += b >> 8;
          lo += b & 255;
          w[i] = (uint32_t)b + 0x80808080u;
        }
        uint32_t dig[4];
        signed_digits(w, dig);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const int col = d * S::NP + 6 * u + j;
          *reinterpret_cast<uint32_t*>(s_img + base + (col >> 3) * S::SBO + (col & 7) * 16) = dig[d];
        }
        hi = __reduce_add_sync(0xffffffffu, hi);  // at most 128 x 2^23
        lo = __reduce_add_sync(0xffffffffu, lo);
        if ((t & 31) == 0) s_sum[t >> 5][6 * u + j] = (long long)hi * 256 + lo;
      }
      if (t == 0)
        a.rec[cell * S::REC + 6 * U + u] = __float_as_uint((float)((double)info.x * V_UNIT * top));
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(a.b + cell * S::TILE_B_BYTES);
    for (int i = t; i < S::TILE_B_BYTES / 16; i += FACTOR_THREADS) dst[i] = reinterpret_cast<const uint4*>(s_img)[i];
    if (t < 6 * U) {
      long long v = 0;
      for (int w = 0; w < FACTOR_THREADS / 32; ++w) v += s_sum[w][t];
      a.rec[cell * S::REC + t] = offset_units(v);
      a.rec[cell * S::REC + 7 * U + t] = __float_as_uint(offset_rest(v));
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------- main kernel ----
struct MmaArgs {
  const float* tiles;
  const double4* anchors;
  const float4* info;
  const float* xy;           // per tile: MMA_XY floats (MmaTiles)
  const unsigned char* b;
  const uint32_t* rec;
  int ntri, ntiles;
  const double* qx;
  const double* qy;
  const double2* rowqz;
  int nqy, nrow, ncol, row0, slab, ncoltiles, nsplit;  // slab: rows from row0 on
  Rot9 R;
  void* out;
  double* part;              // nsplit > 1: [split][q-point of the slab][NACC]
  long part_stride;          // q-points of the slab
  unsigned* err;
};

template <int U, bool PAIRED, typename OUT>
__device__ __forceinline__ void write_pixel(const MmaArgs& a, const double* T, int row, int col) {
  constexpr int NK = PAIRED ? 4 : U;
  OUT* out = reinterpret_cast<OUT*>(a.out);
  const long p = (long)row * a.ncol + col;
  const double qx = a.qx[p], qy = a.qy[p];
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    double sr, si;
    if (PAIRED) {  // blocks 0, 3 from pair 0 (P +- M); blocks 2, 1 from pair 2
      const int pr = (k == 0 || k == 3) ? 0 : 1;
      const double sg = (k == 0 || k == 2) ? 1.0 : -1.0;
      sr = T[4 * pr] + sg * T[4 * pr + 2];
      si = T[4 * pr + 1] + sg * T[4 * pr + 3];
    } else {
      sr = T[2 * k];
      si = T[2 * k + 1];
    }
    const double q2 = rotated_q2(a.R, qx, qy, a.rowqz[(long)row * NK + k]);
    store_ff<OUT>(out, (long)k * a.nqy + p, si / q2, -sr / q2);
  }
}

// One tile's sums for this thread's pixel: read from TMEM (d_tm: the accumulators, this warp's
// lanes), scaled, rotated by the anchor and added to T (stride 128 doubles).
template <int U, bool PAIRED>
__device__ __forceinline__ void add_tile_sums(const MmaArgs& a, uint32_t d_tm, int row, float qx, float qy, float2 e,
                                              const uint32_t* rec, double* T) {
  using S = MmaShape<U>;
  constexpr int NK = PAIRED ? 4 : U;
#pragma unroll
  for (int u = 0; u < U; ++u) {  // one unit = six columns of each slice at a time
    float f[2][6];  // sums with cos, with sin: (n~x, n~y, n~z) Re Z, then Im Z
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      uint32_t d[16];  // two slices at a time
#pragma unroll
      for (int i = 0; i < 2; ++i) tmem_ld8(d_tm + k * S::D_COLS + (2 + i) * S::NP + 6 * u, d + 8 * i);
      tmem_wait_ld<16>(d);
#pragma unroll
      for (int j = 0; j < 6; ++j) f[k][j] = low_sum(d[j], d[8 + j], __uint_as_float(rec[7 * U + 6 * u + j]));
#pragma unroll
      for (int i = 0; i < 2; ++i) tmem_ld8(d_tm + k * S::D_COLS + i * S::NP + 6 * u, d + 8 * i);
      tmem_wait_ld<16>(d);
#pragma unroll
      for (int j = 0; j < 6; ++j) f[k][j] = combined_sum(d[j], d[8 + j], rec[6 * u + j], f[k][j]);
    }
    const float *fc = f[0], *fs = f[1];
    const double2 q = a.rowqz[(long)row * NK + (PAIRED ? 2 * u : u)];
    const float qzr = (float)q.x, qzi = (float)q.y;
    const float scale = __uint_as_float(rec[6 * U + u]);
    const float ex = e.x * scale, ey = e.y * scale;
    if (PAIRED) {
      const float pr = fmaf(qx, fc[0], fmaf(qy, fc[1], -qzr * fs[5]));
      const float pi = fmaf(qx, fs[0], fmaf(qy, fs[1], qzr * fc[5]));
      const float mr = fmaf(-qx, fs[3], fmaf(-qy, fs[4], qzr * fc[2]));
      const float mi = fmaf(qx, fc[3], fmaf(qy, fc[4], qzr * fs[2]));
      T[(4 * u) * 128] += (double)(pr * ex - pi * ey);
      T[(4 * u + 1) * 128] += (double)(pr * ey + pi * ex);
      T[(4 * u + 2) * 128] += (double)(mr * ex - mi * ey);
      T[(4 * u + 3) * 128] += (double)(mr * ey + mi * ex);
    } else {
      float g[3][2];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        g[j][0] = fc[j] - fs[3 + j];
        g[j][1] = fc[3 + j] + fs[j];
      }
      const float sr = fmaf(qx, g[0][0], fmaf(qy, g[1][0], qzr * g[2][0] - qzi * g[2][1]));
      const float si = fmaf(qx, g[0][1], fmaf(qy, g[1][1], qzr * g[2][1] + qzi * g[2][0]));
      T[(2 * u) * 128] += (double)(sr * ex - si * ey);
      T[(2 * u + 1) * 128] += (double)(sr * ey + si * ex);
    }
  }
}

// The q-points next to q = 0: F = S / |q|^2 with S cancelling to |q|^2 of its terms' size over |q|,
// so every rounding counts 1 / (|q| x mesh size) times there, up to 1e-3 of F on fine detectors.
// On a detector's few points of that kind the sums keep the FP32 arithmetic of ff_tri_rows_kernel operation by
// operation, so that both kernels give the same F there.  A point is one of them when some block has
// |q| x (mesh diameter) < NEAR_QD and lies within 2.5 columns (steps of qy) and 2.5 rows of q = 0: a few dozen
// points of a detector at most, none on coarse ones.  Elsewhere (the other such points of a zoomed grid, a single
// column, columns that step along qx) the digits' sums serve, which are the more accurate ones: relative errors
// of a 30 nm mesh at |q| x diameter of 0.02 to 0.2, rms 1.4e-6 against 1.1e-5, below 0.02 1.3e-5 against 4.9e-5.
constexpr double NEAR_QD = 0.2;

template <int U, bool PAIRED>
__device__ __forceinline__ bool near_zero(const MmaArgs& a, int row, int col, double diameter) {
  constexpr int NK = PAIRED ? 4 : U;
  const long p = (long)row * a.ncol + col;
  const int c2 = col + 1 < a.ncol ? col + 1 : col - 1, r2 = row + 1 < a.nrow ? row + 1 : row - 1;
  if (c2 < 0 || r2 < 0) return false;
  const double qx = a.qx[p], qy = a.qy[p], dy = 2.5 * (a.qy[(long)row * a.ncol + c2] - qy);
  if (!(qx * qx + qy * qy < dy * dy)) return false;
  bool near = false;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const double2 q = a.rowqz[(long)row * NK + k], n = a.rowqz[(long)r2 * NK + k];
    const double dz = 2.5 * (n.x - q.x), qz2 = q.x * q.x + q.y * q.y;
    near |= qz2 < dz * dz && (qx * qx + qy * qy + qz2) * diameter * diameter < NEAR_QD * NEAR_QD;
  }
  return near;
}

// The sums of the pixels in list[0 .. count) (columns of `row`) over this CTA's tiles, as the row
// kernel makes them.  A few (pixel, tile) units at a time: all threads make the terms, one lane
// per sum adds a unit's terms in order, one lane per sum folds the units in order.  mem: the tiles'
// shared memory.  Sum n of pixel i goes to out + 8 i + n.
template <int U, bool PAIRED>
__device__ void near_sums(const MmaArgs& a, int row, int t0, int nt, const int* list, int count, float* mem,
                          double* out) {
  using S = MmaShape<U>;
  constexpr int NK = PAIRED ? 4 : U, NF = PAIRED ? 2 : NK, W = 4 + 4 * NF;
  constexpr int UNITS = U == 4 ? 3 : 4;
  static_assert(UNITS * (TILE * W + 8) * 4 <= S::NST * S::STAGE, "the terms take the tiles' place");
  float* parts = mem + UNITS * TILE * W;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = lane < S::NACC ? lane : 0;
  // this lane's sum: factor v[g + fi] times sign times v[oi], in the row kernel's order
  const int g = 4 + 4 * (PAIRED ? n >> 2 : n >> 1);
  int fi[4], oi[4];
  float sg[4];
  if (PAIRED) {  // P.re, P.im, M.re, M.im over (cos, sin, aq cos, aq sin) and (x, y, beta, gamma)
    const int r = n & 3;
    fi[0] = r >> 1;
    oi[0] = r == 0 || r == 3 ? 2 : 3;
    sg[0] = r == 2 ? -1.f : 1.f;
    fi[1] = 2 + (r >> 1);
    oi[1] = r == 0 || r == 3 ? 1 : 0;
    sg[1] = r == 0 ? -1.f : 1.f;
  } else {  // S.re, S.im over the same and (Zr, Zi, DZr, DZi)
    const bool im = n & 1;
    const int f[4] = {im ? 1 : 0, im ? 0 : 1, 2, 3}, o[4] = {2, 3, im ? 1 : 0, im ? 0 : 1};
    for (int i = 0; i < 4; ++i) {
      fi[i] = f[i];
      oi[i] = o[i];
      sg[i] = !im && (i & 1) ? -1.f : 1.f;
    }
  }
  float sum = 0.f, comp = 0.f;  // warp 0, lanes n < NACC: the running sum of the current pixel
  for (int u0 = 0; u0 < count * nt; u0 += UNITS) {
    const int m = min(UNITS, count * nt - u0);
    for (int j = threadIdx.x; j < m * TILE; j += blockDim.x) {
      const int u = u0 + j / TILE, tile = t0 + u % nt;
      const long p = (long)row * a.ncol + list[u / nt];
      const double4 anc = a.anchors[tile];
      const float* tl = a.tiles + (size_t)tile * TILE_FLOATS;
      const float4 t = reinterpret_cast<const float4*>(tl)[j % TILE];
      const float2 bz = reinterpret_cast<const float2*>(tl + 4 * TILE)[j % TILE];
      const float qx = (float)a.qx[p], qy = (float)a.qy[p];
      float tp = fmaf(qx, t.x, qy * t.z);
      if ((float)(anc.w * anc.w) * fmaf(qx, qx, qy * qy) > WIDE_PHASE2) {
        const float tt = tp * INV_TWO_PI_F;
        tp = (tt - round_nearest(tt)) * TWO_PI_F;
      }
      float sn, cs;
      __sincosf(tp, &sn, &cs);
      const float aq = fmaf(qx, t.y, qy * t.w);
      float4* v = reinterpret_cast<float4*>(mem + (size_t)j * W);
      v[0] = make_float4(cs, sn, aq * cs, aq * sn);
      const double cz = anc.z * INV_TWO_PI + (double)bz.x * INV_TWO_PI;
#pragma unroll
      for (int f = 0; f < NF; ++f)
        v[1 + f] = PAIRED ? paired_factor(a.rowqz[(long)row * 4 + 2 * f].x, cz, bz.y)
                          : complex_factor(a.rowqz[(long)row * NK + f], cz, bz.y);
    }
    __syncthreads();
    if (warp < m) {
      const float* v = mem + (size_t)warp * TILE * W;
      float q = 0.f;
#pragma unroll 8
      for (int j = 0; j < TILE; ++j, v += W)
#pragma unroll
        for (int i = 0; i < (PAIRED ? 2 : 4); ++i) q = fmaf(v[g + fi[i]], sg[i] * v[oi[i]], q);
      const int u = u0 + warp;
      const long p = (long)row * a.ncol + list[u / nt];
      const double4 anc = a.anchors[t0 + u % nt];
      const float2 e = anchor_phasor(fma(a.qx[p], anc.x, a.qy[p] * anc.y));
      const float o = __shfl_xor_sync(0xffffffffu, q, 1);  // the other part of the complex sum
      if (lane < S::NACC) parts[8 * warp + lane] = (n & 1) == 0 ? q * e.x - o * e.y : o * e.y + q * e.x;
    }
    __syncthreads();
    if (warp == 0 && lane < S::NACC)
      for (int k = 0; k < m; ++k) {
        float part = parts[8 * k + lane];
        two_sum_fold(sum, part, comp);
        if ((u0 + k) % nt == nt - 1) {
          out[8 * ((u0 + k) / nt) + lane] = (double)sum + (double)comp;
          sum = comp = 0.f;
        }
      }
  }
}

// Every wait is bounded: a thread whose wait gives up (ok = false) waits no more and goes on with
// whatever is there (all addresses stay in range), the CTA writes no result and the error word
// says so.
template <int U, bool PAIRED, typename OUT>
__global__ void __launch_bounds__(MmaShape<U>::THREADS, 1) ff_tri_mma_kernel(MmaArgs a) {
  using S = MmaShape<U>;
  constexpr int SUB = S::SUB;
  extern __shared__ __align__(1024) unsigned char s_mem[];
  __shared__ __align__(8) uint64_t s_full[S::NST];   // a tile has arrived
  __shared__ __align__(8) uint64_t s_ready[SUB];     // a warpgroup's digits are in TMEM
  __shared__ __align__(8) uint64_t s_used[SUB];      // their products are done
  __shared__ __align__(8) uint64_t s_free[S::DBUF];  // an accumulator range has been read
  __shared__ uint32_t s_tmem;
  // the warp's index through a shuffle: known to be uniform, so that the issuing warps' operands
  // are kept in uniform registers
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int wg = warp >> 2, lt = threadIdx.x & 127;  // wg == SUB: the issuing warps
  if (threadIdx.x == 0) {
    for (int i = 0; i < S::NST; ++i) mbar_init(&s_full[i], 1);
    for (int i = 0; i < SUB; ++i) {
      mbar_init(&s_ready[i], 4);
      mbar_init(&s_used[i], 2);
    }
    for (int i = 0; i < S::DBUF; ++i) mbar_init(&s_free[i], 4);
    fence_mbar_init();
  }
  if (warp == SUB * 4) tmem_alloc(&s_tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // TMEM columns: the accumulators, then the warpgroups' digits
  const uint32_t tm = __shfl_sync(0xffffffffu, s_tmem, 0), tm_a = tm + S::DBUF * 2 * S::D_COLS;

  const long item = blockIdx.x;
  const int sp = (int)(item % a.nsplit);
  const int ct = (int)(item / a.nsplit % a.ncoltiles);
  // the last rows first: on a detector they hold the q-points next to q = 0, which take longer
  const int lrow = a.slab - 1 - (int)(item / a.nsplit / a.ncoltiles);
  const int row = a.row0 + lrow;
  const int t0 = (int)((long)sp * a.ntiles / a.nsplit);
  const int nt = (int)((long)(sp + 1) * a.ntiles / a.nsplit) - t0;  // tiles of this CTA (>= 1)
  const int nchunk = MMA_CHUNKS * (nt - 1) + (min(TILE, a.ntri - (t0 + nt - 1) * TILE) + MMA_K - 1) / MMA_K;
  double* sums = reinterpret_cast<double*>(s_mem + S::NST * S::STAGE);
  auto fetch = [&](int i) {  // one thread: tile i of this CTA into its stage
    unsigned char* dst = s_mem + (i % S::NST) * S::STAGE;
    uint64_t* bar = &s_full[i % S::NST];
    mbar_arrive_expect_tx(bar, S::STAGE);
    bulk_g2s(dst, a.b + ((size_t)lrow * a.ntiles + t0 + i) * S::TILE_B_BYTES, S::TILE_B_BYTES, bar);
    bulk_g2s(dst + S::TILE_B_BYTES, a.xy + (size_t)(t0 + i) * MMA_XY, S::XY_BYTES, bar);
    bulk_g2s(dst + S::TILE_B_BYTES + S::XY_BYTES, a.rec + ((size_t)lrow * a.ntiles + t0 + i) * S::REC, S::REC * 4, bar);
  };
  bool ok = true;
  if (wg < SUB) {
    const int col = ct * 128 + lt;
    const bool valid = col < a.ncol;
    const long p = (long)row * a.ncol + col;
    const float qx = valid ? (float)a.qx[p] : 0.f, qy = valid ? (float)a.qy[p] : 0.f;
    const float q2max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaf(qx, qx, qy * qy))));
    double* T = sums + (size_t)wg * S::NACC * 128 + lt;
#pragma unroll
    for (int n = 0; n < S::NACC; ++n) T[n * 128] = 0.0;
    if (threadIdx.x == 0)
      for (int i = 0; i < S::NST && i < nt; ++i) fetch(i);
    const uint32_t lanes = (uint32_t)(lt & 96) << 16;  // this warp's TMEM lanes
    const uint32_t a_tm = tm_a + wg * A_COLS + lanes;
    int n = 0;  // chunks stored
    // The warpgroup that made a tile's last chunk reads the tile's sums back, once that chunk's
    // products are done: the products are issued in order, so the tile's others are done too.
    auto read_back = [&](int i) {
      const int d = i % S::DBUF;
      const double4 anc = a.anchors[t0 + i];
      const float2 e = anchor_phasor(valid ? fma(a.qx[p], anc.x, a.qy[p] * anc.y) : 0.0);
      add_tile_sums<U, PAIRED>(a, tm + d * 2 * S::D_COLS + lanes, row, qx, qy, e,
                               reinterpret_cast<const uint32_t*>(s_mem + (i % S::NST) * S::STAGE + S::TILE_B_BYTES +
                                                                 S::XY_BYTES),
                               T);
      tc_fence_before();
      __syncwarp();
      if ((lt & 31) == 0) mbar_arrive(&s_free[d]);
      // all of the tile's products are done and its record has been read: its stage is free
      wg_sync(wg);
      if (lt == 0 && i + S::NST < nt) {
        fence_proxy_async_smem();
        fetch(i + S::NST);
      }
    };
    auto wait_used = [&]() {  // the products of the chunk stored last
      if (n > 0 && ok) ok = mbar_wait(&s_used[wg], (n - 1) & 1);
      tc_fence_after();
      __syncwarp();
    };
    int unread = -1;  // a tile whose last chunk this warpgroup made
    for (int c = wg; c < nchunk; c += SUB) {
      const int i = c / MMA_CHUNKS, ch = c % MMA_CHUNKS;
      if (ok) ok = mbar_wait(&s_full[i % S::NST], (i / S::NST) & 1);
      const float4* tile = reinterpret_cast<const float4*>(s_mem + (i % S::NST) * S::STAGE + S::TILE_B_BYTES);
      const float4* xy = tile + ch * (MMA_K / 2);
      const float rmax = tile[TILE / 2].x;  // the tile's largest in-plane offset
      const bool wide = rmax * rmax * q2max > WIDE_PHASE2;  // uniform over the warp
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[24];
        if (wide) phasor_digits<true>(xy + 8 * h, qx, qy, w);
        else phasor_digits<false>(xy + 8 * h, qx, qy, w);
        if (h == 0) wait_used();
#pragma unroll
        for (int pl = 0; pl < 6; ++pl) tmem_st4(a_tm + 8 * pl + 4 * h, w + 4 * pl);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if ((lt & 31) == 0) mbar_arrive(&s_ready[wg]);
      ++n;
      // with two accumulator ranges the sums are read one chunk later, when the last products are
      // done without waiting
      if (S::DBUF == 2 && unread >= 0) {
        read_back(unread);
        unread = -1;
      }
      if (ch == MMA_CHUNKS - 1 || c == nchunk - 1) unread = i;
      if (S::DBUF == 1 && unread >= 0) {
        wait_used();
        read_back(unread);
        unread = -1;
      }
    }
    wait_used();  // no arrival is left under way when the block ends
    if (unread >= 0) read_back(unread);
  } else {
    // one warp for the products with cos, one for those with sin (independent accumulators); the
    // whole warp walks the chunks so that the operands stay in uniform registers
    const int t = warp - SUB * 4;
    int k = 0, use = 0, left = nchunk;  // warpgroup of the chunk, its chunk number
    for (int i = 0; i < nt; ++i) {
      const int d = i % S::DBUF;
      if (ok) ok = mbar_wait(&s_full[i % S::NST], (i / S::NST) & 1);
      if (i >= S::DBUF && ok) ok = mbar_wait(&s_free[d], (i / S::DBUF - 1) & 1);
      const uint32_t dc = tm + (2 * d + t) * S::D_COLS;
      uint64_t bd = smem_desc(smem_addr(s_mem + (i % S::NST) * S::STAGE), S::LBO, S::SBO);
      const int nch = min(MMA_CHUNKS, left);
      left -= nch;
      for (int ch = 0; ch < nch; ++ch) {
        if (ok) ok = mbar_wait(&s_ready[k], use & 1);
        tc_fence_after();
        __syncwarp();
        const uint32_t av = tm_a + k * A_COLS + 24 * t;
        if (elect_one()) {
          mma_s8_ts(dc, av, bd, idesc_s8(4 * S::NP), ch > 0);
          mma_s8_ts(dc + S::NP, av + 8, bd, idesc_s8(3 * S::NP), 1);
          mma_s8_ts(dc + 2 * S::NP, av + 16, bd, idesc_s8(2 * S::NP), 1);
          mma_commit(&s_used[k]);
        }
        __syncwarp();
        bd += S::CHUNK_BYTES >> 4;
        if (++k == SUB) {
          k = 0;
          ++use;
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  const bool failed = __syncthreads_or(!ok);
  tc_fence_after();
  if (failed) {
    if (threadIdx.x == 0) {  // what is still in flight is waited for (bounded)
      atomicOr(a.err, (unsigned)DEV_ERR_WAIT_TIMEOUT);
      for (int i = nt > S::NST ? nt - S::NST : 0; i < nt; ++i) mbar_wait(&s_full[i % S::NST], (i / S::NST) & 1);
      for (int k = 0; k < SUB && k < nchunk; ++k) mbar_wait(&s_used[k], ((nchunk - 1 - k) / SUB) & 1);
    }
    __syncthreads();
  } else {
    // which of the CTA's pixels lie next to q = 0 (the mesh's diameter is bounded over its tiles)
    __shared__ int s_near[128], s_nnear;
    const int col = ct * 128 + lt;
    bool near = false;
    if (wg == 0 && col < a.ncol && near_zero<U, PAIRED>(a, row, col, 0.0)) {
      double diameter = 0.0;
      const double4 c0 = a.anchors[0];
      for (int i = 0; i < a.ntiles; ++i) {
        const double4 c = a.anchors[i];
        const float4 f = a.info[i];
        const double dx = TWO_PI * (c.x - c0.x), dy = TWO_PI * (c.y - c0.y), dz = c.z - c0.z;
        diameter = fmax(diameter, sqrt(dx * dx + dy * dy + dz * dz) + c.w + (double)fmaxf(-f.y, f.z));
      }
      near = near_zero<U, PAIRED>(a, row, col, diameter);
    }
    if (__syncthreads_or(near)) {
      if (threadIdx.x == 0) s_nnear = 0;
      __syncthreads();
      if (near) s_near[atomicAdd(&s_nnear, 1)] = col;  // the order does not matter
      __syncthreads();
      double* exactly = sums + (size_t)SUB * S::NACC * 128;
      near_sums<U, PAIRED>(a, row, t0, nt, s_near, s_nnear, reinterpret_cast<float*>(s_mem), exactly);
      __syncthreads();
    }
    if (wg == 0 && col < a.ncol) {
      double T[S::NACC];
#pragma unroll
      for (int n = 0; n < S::NACC; ++n) {
        T[n] = 0.0;
        for (int w = 0; w < SUB; ++w) T[n] += sums[(size_t)(w * S::NACC + n) * 128 + lt];
      }
      if (near)
        for (int i = 0; i < s_nnear; ++i)
          if (s_near[i] == col)
            for (int n = 0; n < S::NACC; ++n) T[n] = sums[(size_t)SUB * S::NACC * 128 + 8 * i + n];
      if (a.nsplit > 1) {
        double* dst = a.part + ((size_t)sp * a.part_stride + (long)lrow * a.ncol + col) * S::NACC;
#pragma unroll
        for (int n = 0; n < S::NACC; ++n) dst[n] = T[n];
      } else {
        write_pixel<U, PAIRED, OUT>(a, T, row, col);
      }
    }
  }
  if (warp == SUB * 4) tmem_free(tm, 512);
}

// Adds the splits' sums in a fixed order and writes the form factor.
template <int U, bool PAIRED, typename OUT>
__global__ void __launch_bounds__(128) ff_tri_mma_sum_kernel(MmaArgs a) {
  using S = MmaShape<U>;
  const long i = (long)blockIdx.x * 128 + threadIdx.x;
  if (i >= a.part_stride) return;
  double T[S::NACC];
#pragma unroll
  for (int n = 0; n < S::NACC; ++n) T[n] = 0.0;
  for (int sp = 0; sp < a.nsplit; ++sp) {
    const double* src = a.part + ((size_t)sp * a.part_stride + i) * S::NACC;
#pragma unroll
    for (int n = 0; n < S::NACC; ++n) T[n] += src[n];
  }
  write_pixel<U, PAIRED, OUT>(a, T, a.row0 + (int)(i / a.ncol), (int)(i % a.ncol));
}

// -------------------------------------------------------------------- host ----
constexpr size_t SLAB_BYTES = (size_t)1 << 30;  // row factors held at a time
constexpr size_t PART_BYTES = (size_t)256 << 20;  // split partial sums

template <int U, bool PAIRED, typename OUT>
static int run(hgx_ctx c, hgx_qgrid g, const MmaTiles& t, const Rot9& R, void* out) {
  using S = MmaShape<U>;
  cudaStream_t st = c->stream;
  const size_t row_bytes = (size_t)t.ntiles * (S::TILE_B_BYTES + S::REC * 4);
  const int ncoltiles = (g->ncol + 127) / 128;
  const long wave = c->sm_count;  // items running at a time
  long rows = std::min<long>(g->nrow, std::max<size_t>(1, SLAB_BYTES / row_bytes));
  int nsplit = 1;
  if (rows < g->nrow) {
    // several slabs: whole waves of items each, so that none ends with a nearly empty one
    const long full = rows * ncoltiles / wave * wave / ncoltiles;
    if (full > 0) rows = full;
  } else {
    // few items: the tiles are split over CTAs where that fills the last wave better; an item's own
    // cost (its start, first fetch and end) is about a tile's, and so is adding the splits' sums
    const long items = rows * ncoltiles;
    const size_t part = (size_t)rows * g->ncol * S::NACC * sizeof(double);
    double best = 0.0;
    for (int k = 1; k <= t.ntiles && k <= 32 && (k == 1 || k * part <= PART_BYTES); ++k) {
      const double cost = (double)((items * k + wave - 1) / wave) * ((t.ntiles + k - 1) / k + 1.0) + (k > 1);
      if (k == 1 || cost < best) {
        best = cost;
        nsplit = k;
      }
    }
  }
  const size_t b_bytes = (size_t)rows * t.ntiles * S::TILE_B_BYTES;
  const size_t rec_bytes = (size_t)rows * t.ntiles * S::REC * 4;
  const size_t rec_pad = (rec_bytes + 255) & ~(size_t)255;
  const size_t part_bytes = nsplit > 1 ? (size_t)nsplit * rows * g->ncol * S::NACC * sizeof(double) : 0;
  // nothing is allocated while the stream is captured (the FP32 kernel then takes the call), and a
  // block that a graph holds stays allocated
  if (is_capturing(st)) {
    if (c->factors.bytes < b_bytes + rec_pad + part_bytes) return HGX_ERR_NO_MEMORY;
    c->factors.captured = true;
  }
  HGX_TRY(c->factors.reserve(b_bytes + rec_pad + part_bytes));
  unsigned char* base = reinterpret_cast<unsigned char*>(c->factors.p);
  HGX_CUDA(cudaFuncSetAttribute(ff_tri_mma_kernel<U, PAIRED, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                S::SMEM));
  HGX_CUDA(cudaFuncSetAttribute(ff_row_factor_kernel<U, PAIRED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                S::TILE_B_BYTES));
  for (int row0 = 0; row0 < g->nrow; row0 += (int)rows) {
    const int n = (int)std::min<long>(rows, g->nrow - row0);
    FactorArgs f{t.tiles, t.anchors, t.info, g->rowqz, t.ntiles, row0, n, base,
                 reinterpret_cast<uint32_t*>(base + b_bytes)};
    const int groups = std::min(n, std::max(1, 8 * c->sm_count / t.ntiles));
    ff_row_factor_kernel<U, PAIRED><<<dim3(t.ntiles, groups), FACTOR_THREADS, S::TILE_B_BYTES, st>>>(f);
    MmaArgs a{t.tiles, t.anchors, t.info, t.xy, f.b, f.rec, t.ntri, t.ntiles, g->qx, g->qy, g->rowqz, g->nqy, g->nrow, g->ncol, row0, n,
              ncoltiles, nsplit, R, out,
              reinterpret_cast<double*>(base + b_bytes + rec_pad), (long)n * g->ncol, c->d_err};
    ff_tri_mma_kernel<U, PAIRED, OUT><<<(unsigned)((long)n * ncoltiles * nsplit), S::THREADS, S::SMEM, st>>>(a);
    if (nsplit > 1)
      ff_tri_mma_sum_kernel<U, PAIRED, OUT><<<(unsigned)((a.part_stride + 127) / 128), 128, 0, st>>>(a);
    HGX_CUDA(cudaGetLastError());
  }
  return HGX_OK;
}

int ff_rows_mma(hgx_ctx c, hgx_qgrid g, const MmaTiles& t, const Rot9& R, void* out, int ff_type) {
  const bool c64 = ff_type == HGX_C64;
  if (g->mode == 1) return c64 ? run<2, true, float2>(c, g, t, R, out) : run<2, true, double2>(c, g, t, R, out);
  if (g->nk == 4) return c64 ? run<4, false, float2>(c, g, t, R, out) : run<4, false, double2>(c, g, t, R, out);
  return c64 ? run<1, false, float2>(c, g, t, R, out) : run<1, false, double2>(c, g, t, R, out);
}

}  // namespace hgx
