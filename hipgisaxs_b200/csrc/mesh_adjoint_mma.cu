// The mesh adjoint's backward pass (mesh_adjoint.cu) with its sums over pixels on the tensor cores.
//
// With the notation there (row phasors Z_0 = x + i y of the pair 03, Z_2 of the pair 21; seeds P, M of
// a pair rotated by the tile's anchor phasor; E = e^{i q_par.d} of a (pixel, triangle)), the gradients
// of a triangle over the pixels of one detector row need, per pair, only the moments
//   Re X_P, Im X_M                 with weights qx, qy,
//   Im X_P, Re X_M                 with weights 1, qx^2, qx qy, qy^2,     X_H^m = sum_p m E H,
// because P enters times x and M times i y:
//   g_n  += (Re X_P^x x - Im X_M^x y, Re X_P^y x - Im X_M^y y, qz (Re X_M^1 x - Im X_P^1 y)),
//   g_c  -= (n~x I^xx + n~y I^xy + n~z J^x, n~x I^xy + n~y I^yy + n~z J^y, n~x J^x + n~y J^y + n~z K),
//   I^m = Im X_P^m x + Re X_M^m y,  J^m = qz (Im X_M^m x + Re X_P^m y),  K = qz^2 I^1.
// So a row's sums are a matrix product of the phasors (c, s of E: lanes = triangles, K = pixels) with
// 24 real columns for c and 24 for s, Re X = sum c Hr - s Hi and Im X = sum c Hi + s Hr, which add up
// in the same accumulators.  Digits, accumulation and roles of the warps are those of ff_tri_mma.cu
// with pixels and triangles exchanged: a CTA owns 128 triangles (a quarter of a tile) and a range of
// detector rows, cut into items of up to 256 pixels of a row; five warpgroups make the phasors'
// digits, one warp fetches the items and issues the products, and the warpgroup that made an item's
// last digits reads its sums back, applies the row phasors and adds to FP64 sums.
//
// The seeds have four digits, scaled by the largest modulus of their column in the item: a vertex
// gradient is the small difference of its triangles' sums, so what an item rounds off its weak
// pixels shows.  Vertex gradients of 80 meshes (320 to 5,120 faces, radius 3 to 40 nm) against FP64,
// geometric mean of the error over the FP32 kernel's: 0.74, never above 1e-6 where it is larger;
// with three digits 0.95, but up to 2.4 times (4e-6) on fine meshes of 20 to 40 nm, and 6% faster.
//
// Bound as ff_tri_mma_kernel by the SFU and issue of the digit makers, plus a tenth for reading the
// sums back.  512 x 512 pixels x 20,000 triangles: 4.25 ms and 0.82 ms for the seeds' digits (2.5 GB,
// 3.1 TB/s); the FP32 kernel of mesh_adjoint.cu (80 FP32 operations per pixel and triangle) 11.3 ms.
// A stage is refilled by the issuing warp as soon as its products are done; refilled after the
// read-back instead, the same two stages gave 4.8 ms.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "ff_tri_digits.cuh"
#include "mesh_adjoint.cuh"
#include "ptx.cuh"
#include "tc05.cuh"

namespace hgx {

constexpr int BWM_SUB = 5;
constexpr int BWM_THREADS = BWM_SUB * 128 + 32;
constexpr int BWM_NP = 32;                    // columns per digit slice: 16 per pair, 12 used
constexpr int BWM_ND = 4;                     // seed digits
constexpr int BWM_LBO = BWM_ND * BWM_NP / 8 * 128;
constexpr int BWM_TRIG = 2 * BWM_LBO;         // seed digits of 32 pixels for cos; the same for sin follow
constexpr int BWM_CHUNK = 2 * BWM_TRIG;
constexpr int BWM_MAX_CHUNKS = 8;             // 32-pixel chunks per item
constexpr int BWM_REC = 72;                   // words per (item, tile): 24 offsets, 24 scales, 24 offsets' rests
constexpr int BWM_STAGE = BWM_MAX_CHUNKS * (BWM_CHUNK + 256) + 16;
constexpr int BWM_NST = 2;
constexpr int BWM_SUMS = BWM_SUB * 6 * 128 * 8;
constexpr int BWM_NREC = 4;                   // items whose records are held
constexpr int BWM_SMEM = BWM_NST * BWM_STAGE + BWM_NREC * BWM_REC * 4 + BWM_SUMS;
constexpr int BWM_D = BWM_ND * BWM_NP;        // accumulator columns, two ranges

// Column j of a pair's 12: weight and which number of (P, M).
//   0 ReP qx, 1 ImM qx, 2 ReP qy, 3 ImM qy, 4 ImP, 5 ReM, 6 ImP qx^2, 7 ReM, 8 ImP qx qy, 9 ReM, 10 ImP qy^2, 11 ReM
__device__ __forceinline__ float moment(int j, float qx, float qy) {
  return j < 2 ? qx : j < 4 ? qy : j < 6 ? 1.f : j < 8 ? qx * qx : j < 10 ? qx * qy : qy * qy;
}

// |x + i y|, also where the squares leave FP32's range.
__device__ __forceinline__ float modulus(float x, float y) {
  const float m = fmaxf(fabsf(x), fabsf(y));
  return m > 1e-15f && m < 1e15f ? sqrtf(x * x + y * y) : hypotf(x, y);
}

// Per item (one CTA): the in-plane q of its pixels as the digit makers read them (pairs, then the
// largest |q_par|), and the largest modulus of every seed column.
__global__ void __launch_bounds__(256) bwm_item_kernel(BwmArgs a, int row0) {
  __shared__ float s_max[8][25];
  const int row = row0 + blockIdx.y, item = blockIdx.y * a.nch + blockIdx.x, w = a.nck * 32;
  const int i = threadIdx.x, col = blockIdx.x * w + i;
  const bool in = i < w && col < a.ncol;
  const long p = (long)row * a.ncol + col;
  const float qx = in ? (float)a.qx[p] : 0.f, qy = in ? (float)a.qy[p] : 0.f;
  float v[25];
  const float4 none = make_float4(0, 0, 0, 0), s[2] = {in ? a.seeds[2 * p] : none, in ? a.seeds[2 * p + 1] : none};
#pragma unroll
  for (int pr = 0; pr < 2; ++pr) {
    float mp = modulus(s[pr].x, s[pr].y), mm = modulus(s[pr].z, s[pr].w);
    if (!isfinite(mp)) mp = INFINITY;  // the gradient is then not finite either
    if (!isfinite(mm)) mm = INFINITY;
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      const float m = fabsf(moment(j, qx, qy));
      v[12 * pr + j] = (j & 1) == 0 ? (mp == INFINITY ? mp : m * mp) : (mm == INFINITY ? mm : m * mm);
    }
  }
  v[24] = sqrtf(qx * qx + qy * qy);
  if (i < w) {
    float* xy = a.xy + (size_t)item * (w * 2 + 4) + (i >> 1) * 4 + (i & 1);
    xy[0] = qx;
    xy[2] = qy;
  }
#pragma unroll
  for (int j = 0; j < 25; ++j) {
    const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v[j])));
    if ((i & 31) == 0) s_max[i >> 5][j] = m;
  }
  __syncthreads();
  if (i < 25) {
    float m = s_max[0][i];
    for (int k = 1; k < 8; ++k) m = fmaxf(m, s_max[k][i]);
    if (i < 24) a.colmax[(size_t)item * 24 + i] = fmaxf(m, 0x1p-124f);  // keeps both scales in range
    else {
      float* e = a.xy + (size_t)item * (w * 2 + 4) + w * 2;
      e[0] = m;
      e[1] = e[2] = e[3] = 0.f;
    }
  }
}

// The seed digits of one item for one tile: a thread does four pixels of one pair for cos or sin.  They
// are put together in shared memory, where a gap behind every half and chunk spreads the
// eight half chunks that a warp writes to over the banks.
constexpr int BWM_IMG_LBO = BWM_LBO + 16;
constexpr int BWM_IMG_CHUNK = 4 * BWM_IMG_LBO + 96;

__global__ void __launch_bounds__(256) bwm_seed_kernel(BwmArgs a, int row0) {
  extern __shared__ __align__(16) unsigned char s_img[];
  __shared__ long long s_sum[8][12];
  const int tile = blockIdx.x, item = blockIdx.y, t = threadIdx.x & 63, pr = (threadIdx.x >> 6) & 1;
  const int trig = threadIdx.x >> 7;
  const int row = row0 + item / a.nch, chunk = item % a.nch, w = a.nck * 32;
  const double4 anc = a.anchors[tile];
  float q[4][2], h[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = 4 * t + i, col = chunk * w + k;
    const bool in = k < w && col < a.ncol;
    const long p = (long)row * a.ncol + col;
    const double qx = in ? a.qx[p] : 0.0, qy = in ? a.qy[p] : 0.0;
    float4 v = in ? a.seeds[2 * p + pr] : make_float4(0, 0, 0, 0);
    const float2 e = anchor_phasor(fma(qx, anc.x, qy * anc.y));
    q[i][0] = (float)qx;
    q[i][1] = (float)qy;
    rotate_pair(v.x, v.y, e);
    rotate_pair(v.z, v.w, e);
    // c takes Pr, Mi (weights qx, qy) or Pi, Mr; s takes -Pi, Mr or Pr, -Mi
    h[i][0] = trig ? -v.y : v.x;
    h[i][1] = trig ? v.z : v.w;
    h[i][2] = trig ? v.x : v.y;
    h[i][3] = trig ? -v.w : v.z;
  }
  unsigned char* img = s_img + (t >> 3) * BWM_IMG_CHUNK + (2 * trig + ((t >> 2) & 1)) * BWM_IMG_LBO + (t & 3) * 4;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    uint32_t x[4], dig[BWM_ND] = {0, 0, 0, 0};
    if (j < 12) {
      // two factors where one would leave FP32's range
      const float top = a.colmax[(size_t)item * 24 + 12 * pr + j], up = top < 0x1p-60f ? 0x1p64f : 1.f;
      const float sc = (float)(B_SCALE / ((double)top * (double)up));
      int hi = 0, lo = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int b = __float2int_rn(moment(j, q[i][0], q[i][1]) * h[i][(j < 4 ? 0 : 2) + (j & 1)] * up * sc);
        hi += b >> 8;
        lo += b & 255;
        x[i] = (uint32_t)b + 0x80808080u;
      }
      signed_digits(x, dig);
      hi = __reduce_add_sync(0xffffffffu, hi);
      lo = __reduce_add_sync(0xffffffffu, lo);
      if ((t & 31) == 0) s_sum[threadIdx.x >> 5][j] = (long long)hi * 256 + lo;
    }
    if (t < a.nck * 8)
#pragma unroll
      for (int d = 0; d < BWM_ND; ++d) {
        const int col = d * BWM_NP + 16 * pr + j;
        *reinterpret_cast<uint32_t*>(img + (col >> 3) * 128 + (col & 7) * 16) = dig[d];
      }
  }
  __syncthreads();
  const size_t cell = (size_t)item * a.ntiles + tile;
  uint4* dst = reinterpret_cast<uint4*>(a.b + cell * a.nck * BWM_CHUNK);
  constexpr int HALF = BWM_LBO / 16;
  for (int i = threadIdx.x; i < a.nck * 4 * HALF; i += 256)
    dst[i] = *reinterpret_cast<const uint4*>(s_img + i / (4 * HALF) * BWM_IMG_CHUNK + (i / HALF & 3) * BWM_IMG_LBO +
                                             i % HALF * 16);
  if (threadIdx.x < 24) {
    const int c = threadIdx.x, w0 = c / 12 * 2, j = c % 12;
    const long long off = s_sum[w0][j] + s_sum[w0 + 1][j] + s_sum[w0 + 4][j] + s_sum[w0 + 5][j];
    const float top = a.colmax[(size_t)item * 24 + c];
    uint32_t* rec = a.rec + cell * BWM_REC + c;
    rec[0] = offset_units(off);
    rec[24] = __float_as_uint(top == INFINITY ? NAN : (float)((double)top * V_UNIT));
    rec[48] = __float_as_uint(offset_rest(off));
  }
}

// One item's sums for this thread's triangle, added to g (6 FP64 sums, stride 128).
__device__ __forceinline__ void bwm_add(uint32_t d_tm, const uint32_t* rec, double qz0, double qz2, double cz, float nx,
                                        float ny, float nz, double* g) {
  float gn[3] = {0.f, 0.f, 0.f}, gc[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int pr = 0; pr < 2; ++pr) {
    float f[12];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // eight columns of each slice, four used of the second
      uint32_t d[8 * BWM_ND];
#pragma unroll
      for (int i = 0; i < BWM_ND; ++i) tmem_ld8(d_tm + i * BWM_NP + 16 * pr + 8 * h, d + 8 * i);
      tmem_wait_ld<8 * BWM_ND>(d);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = 12 * pr + 8 * h + j;
        if (8 * h + j < 12) {
          f[8 * h + j] = combined_sum(d[j], d[8 + j], rec[c], low_sum(d[16 + j], d[24 + j], __uint_as_float(rec[48 + c]))) *
                         __uint_as_float(rec[24 + c]);
        }
      }
    }
    const double qz = pr ? qz2 : qz0;
    double u = qz * cz;
    u -= rint(u);
    float x, y;
    sincospif((float)(2.0 * u), &y, &x);
    const float q = (float)qz;
    gn[0] += f[0] * x - f[1] * y;
    gn[1] += f[2] * x - f[3] * y;
    gn[2] += q * (f[5] * x - f[4] * y);
    const float jx = q * (f[1] * x + f[0] * y), jy = q * (f[3] * x + f[2] * y), kk = q * q * (f[4] * x + f[5] * y);
    const float ixx = f[6] * x + f[7] * y, ixy = f[8] * x + f[9] * y, iyy = f[10] * x + f[11] * y;
    gc[0] += nx * ixx + ny * ixy + nz * jx;
    gc[1] += nx * ixy + ny * iyy + nz * jy;
    gc[2] += nx * jx + ny * jy + nz * kk;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g[k * 128] += (double)gn[k];
    g[(3 + k) * 128] -= (double)gc[k];
  }
}

// Every wait is bounded, as in ff_tri_mma_kernel: a thread whose wait gives up goes on without
// waiting (all addresses stay in range) and the error word says so.
__global__ void __launch_bounds__(BWM_THREADS, 1) bwm_kernel(BwmArgs a, int row0, int nrows) {
  constexpr int SUB = BWM_SUB, NST = BWM_NST;
  extern __shared__ __align__(1024) unsigned char s_mem[];
  __shared__ __align__(8) uint64_t s_full[NST], s_ready[SUB], s_used[SUB], s_free[2], s_done;
  __shared__ uint32_t s_tmem;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int wg = warp >> 2, lt = threadIdx.x & 127;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NST; ++i) mbar_init(&s_full[i], 1);
    for (int i = 0; i < SUB; ++i) {
      mbar_init(&s_ready[i], 4);
      mbar_init(&s_used[i], 1);
    }
    mbar_init(&s_done, 1);
    mbar_init(&s_free[0], 4);
    mbar_init(&s_free[1], 4);
    fence_mbar_init();
  }
  if (warp == SUB * 4) tmem_alloc(&s_tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = __shfl_sync(0xffffffffu, s_tmem, 0), tm_a = tm + 2 * BWM_D;

  // triangles quarter * 128 .. of a tile, rows ra .. rb - 1 of the slab
  const int tile = blockIdx.x >> 2, quarter = blockIdx.x & 3;
  const int ra = (int)((long)blockIdx.y * nrows / gridDim.y), rb = (int)((long)(blockIdx.y + 1) * nrows / gridDim.y);
  const int item0 = ra * a.nch, ni = (rb - ra) * a.nch, nck = a.nck;
  const int b_bytes = nck * BWM_CHUNK, xy_bytes = nck * 256 + 16;
  uint32_t* s_rec = reinterpret_cast<uint32_t*>(s_mem + NST * BWM_STAGE);
  double* s_sums = reinterpret_cast<double*>(s_rec + BWM_NREC * BWM_REC);
  auto fetch = [&](int i) {  // one thread: item i into its stage
    unsigned char* dst = s_mem + (i % NST) * BWM_STAGE;
    uint64_t* bar = &s_full[i % NST];
    const size_t cell = (size_t)(item0 + i) * a.ntiles + tile;
    mbar_arrive_expect_tx(bar, b_bytes + xy_bytes + BWM_REC * 4);
    bulk_g2s(dst, a.b + cell * b_bytes, b_bytes, bar);
    bulk_g2s(dst + b_bytes, a.xy + (size_t)(item0 + i) * (nck * 64 + 4), xy_bytes, bar);
    bulk_g2s(s_rec + (i % BWM_NREC) * BWM_REC, a.rec + cell * BWM_REC, BWM_REC * 4, bar);
  };
  bool ok = true;
  if (wg < SUB) {
    const float* tl = a.tiles + (size_t)tile * TILE_FLOATS;
    const float4 A = reinterpret_cast<const float4*>(tl)[quarter * 128 + lt];  // dx, n~x, dy, n~y
    const float2 B = reinterpret_cast<const float2*>(tl + 4 * TILE)[quarter * 128 + lt];
    const float d2max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaf(A.x, A.x, A.z * A.z))));
    const double cz = a.anchors[tile].z * INV_TWO_PI + (double)B.x * INV_TWO_PI;
    double* g = s_sums + (size_t)wg * 6 * 128 + lt;
#pragma unroll
    for (int k = 0; k < 6; ++k) g[k * 128] = 0.0;
    const uint32_t lanes = (uint32_t)(lt & 96) << 16;
    const uint32_t a_tm = tm_a + wg * A_COLS + lanes;
    int n = 0;
    auto read_back = [&](int i) {
      const int row = row0 + ra + i / a.nch;
      const double qz0 = a.rowqz[4L * row].x, qz2 = a.rowqz[4L * row + 2].x;
      bwm_add(tm + (i & 1) * BWM_D + lanes, s_rec + (i % BWM_NREC) * BWM_REC, qz0, qz2, cz, A.y, A.w, B.y, g);
      tc_fence_before();
      __syncwarp();
      if ((lt & 31) == 0) mbar_arrive(&s_free[i & 1]);
    };
    auto wait_used = [&]() {
      if (n > 0 && ok) ok = mbar_wait(&s_used[wg], (n - 1) & 1);
      tc_fence_after();
      __syncwarp();
    };
    int unread = -1;
    for (int c = wg; c < ni * nck; c += SUB) {
      const int i = c / nck, ch = c - i * nck;
      if (ok) ok = mbar_wait(&s_full[i % NST], (i / NST) & 1);
      const float4* px = reinterpret_cast<const float4*>(s_mem + (i % NST) * BWM_STAGE + b_bytes);
      const float qmax = px[nck * 16].x;
      const bool wide = qmax * qmax * d2max > WIDE_PHASE2;
      px += ch * (MMA_K / 2);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[24];
        if (wide) phasor_digits<true>(px + 8 * h, A.x, A.z, w);
        else phasor_digits<false>(px + 8 * h, A.x, A.z, w);
        if (h == 0) wait_used();
#pragma unroll
        for (int pl = 0; pl < 6; ++pl) tmem_st4(a_tm + 8 * pl + 4 * h, w + 4 * pl);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if ((lt & 31) == 0) mbar_arrive(&s_ready[wg]);
      ++n;
      if (unread >= 0) {  // an item has at least SUB chunks: this one belongs to the item after it
        read_back(unread);
        unread = -1;
      }
      if (ch == nck - 1) unread = i;
    }
    wait_used();  // no arrival is left under way when the block ends
    if (unread >= 0) read_back(unread);
  } else {
    int k = 0, use = 0;
    if (elect_one())
      for (int i = 0; i < NST && i < ni; ++i) fetch(i);
    __syncwarp();
    for (int i = 0; i < ni; ++i) {
      if (ok) ok = mbar_wait(&s_full[i % NST], (i / NST) & 1);
      if (i >= 2 && ok) ok = mbar_wait(&s_free[i & 1], (i / 2 - 1) & 1);
      const uint32_t dc = tm + (i & 1) * BWM_D;
      uint64_t bd = smem_desc(smem_addr(s_mem + (i % NST) * BWM_STAGE), BWM_LBO, 128);
      for (int ch = 0; ch < nck; ++ch) {
        if (ok) ok = mbar_wait(&s_ready[k], use & 1);
        tc_fence_after();
        __syncwarp();
        const uint32_t av = tm_a + k * A_COLS;
        if (elect_one()) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const uint64_t b = bd + t * (BWM_TRIG >> 4);
            mma_s8_ts(dc, av + 24 * t, b, idesc_s8(4 * BWM_NP), t > 0 || ch > 0);
            mma_s8_ts(dc + BWM_NP, av + 24 * t + 8, b, idesc_s8(3 * BWM_NP), 1);
            mma_s8_ts(dc + 2 * BWM_NP, av + 24 * t + 16, b, idesc_s8(2 * BWM_NP), 1);
          }
          mma_commit(&s_used[k]);
          if (ch == nck - 1 && i + 1 < ni) mma_commit(&s_done);  // waited for below, in the next item
        }
        __syncwarp();
        // Two chunks on, the last item's products are done and its pixels were read before: its
        // stage takes the item after this one.  (Its record stays until s_free above.)
        if (ch == 1 && i > 0) {
          if (ok) ok = mbar_wait(&s_done, (i - 1) & 1);
          if (i - 1 + NST < ni && elect_one()) {
            fence_proxy_async_smem();
            fetch(i - 1 + NST);
          }
          __syncwarp();
        }
        bd += BWM_CHUNK >> 4;
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
    if (threadIdx.x == 0) {
      atomicOr(a.err, (unsigned)DEV_ERR_WAIT_TIMEOUT);
      for (int i = ni > NST ? ni - NST : 0; i < ni; ++i) mbar_wait(&s_full[i % NST], (i / NST) & 1);
      for (int k = 0; k < SUB; ++k) mbar_wait(&s_used[k], ((ni * nck - 1 - k) / SUB) & 1);
      if (ni > 1) mbar_wait(&s_done, (ni - 2) & 1);
    }
    __syncthreads();
  } else if (wg == 0) {
    const int t = a.perm[(size_t)tile * TILE + quarter * 128 + lt];
    if (t >= 0) {
      const double* sums = s_sums + lt;
      double* dst = a.partial + ((size_t)blockIdx.y * a.ntri + t) * 6;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        double v = 0.0;
        for (int w = 0; w < SUB; ++w) v += sums[(w * 6 + k) * 128];
        dst[k] = row0 ? dst[k] + v : v;  // a later slab adds to the earlier ones' sums
      }
    }
  }
  if (warp == SUB * 4) tmem_free(tm, 512);
}

// -------------------------------------------------------------------- host ----
constexpr size_t BWM_SLAB_BYTES = (size_t)1 << 30;  // seed digits held at a time
constexpr size_t BWM_PART_BYTES = (size_t)64 << 20;  // partial sums (one row range's at least)

// Grids of up to 128 columns stay with the FP32 kernel: an item needs a chunk per warpgroup.  From 129
// on this pass is the faster one at every size tried (whole call, both with the same forward: 130 x 2 x
// 20 faces 0.150 against 0.156 ms, 130 x 64 x 1,280 0.211 / 0.239, 256 x 64 x 5,120 0.40 / 0.52,
// 130 x 300 x 5,120 0.93 / 1.08, 512 x 512 x 5,120 2.39 / 4.10).
BwmPlan bwm_plan(hgx_ctx c, hgx_qgrid g, int ntiles, int ntri) {
  BwmPlan p{};
  // items of equal width, at least BWM_SUB chunks each
  if (g->ncol <= 32 * (BWM_SUB - 1)) return p;
  p.nch = (g->ncol + 32 * BWM_MAX_CHUNKS - 1) / (32 * BWM_MAX_CHUNKS);
  p.nck = (g->ncol + 32 * p.nch - 1) / (32 * p.nch);
  const size_t row = (size_t)p.nch * (ntiles * ((size_t)p.nck * BWM_CHUNK + BWM_REC * 4) + p.nck * 256 + 16 + 24 * 4);
  p.rows = (int)std::max<size_t>(1, std::min<size_t>(g->nrow, BWM_SLAB_BYTES / row));
  p.slabs = (g->nrow + p.rows - 1) / p.rows;
  p.rows = (g->nrow + p.slabs - 1) / p.slabs;  // slabs of equal size
  // row ranges per group of triangles: whole waves of CTAs, a CTA's own cost about one item.  The slabs
  // share the ranges' partial sums, so that these do not grow with the number of slabs (itself
  // proportional to pixels x triangles).
  const int groups = (ntri + 127) / 128;
  double best = 0.0;
  for (int k = 1; k <= p.rows && k <= 64 && (k == 1 || k * sizeof(double) * 6 * (size_t)ntri <= BWM_PART_BYTES); ++k) {
    const double cost = (double)((groups * (long)k + c->sm_count - 1) / c->sm_count) *
                        ((double)((p.rows + k - 1) / k) * p.nch + 1.5);
    if (k == 1 || cost < best) {
      best = cost;
      p.splits = k;
    }
  }
  return p;
}

int bwm_run(hgx_ctx c, const BwmPlan& p, BwmArgs a) {
  static_assert(BWM_SMEM <= 227 * 1024 && 2 * BWM_D + BWM_SUB * A_COLS <= 512, "shared memory and TMEM of one SM");
  cudaStream_t st = c->stream;
  a.nch = p.nch;
  a.nck = p.nck;
  const size_t items = (size_t)p.rows * p.nch;
  auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
  const size_t nb = up(items * a.ntiles * p.nck * BWM_CHUNK), nr = up(items * a.ntiles * BWM_REC * 4),
               nx = up(items * (p.nck * 256 + 16)), nm = up(items * 24 * 4);
  HGX_TRY(c->factors.reserve(nb + nr + nx + nm));
  unsigned char* base = reinterpret_cast<unsigned char*>(c->factors.p);
  a.b = base;
  a.rec = reinterpret_cast<uint32_t*>(base + nb);
  a.xy = reinterpret_cast<float*>(base + nb + nr);
  a.colmax = reinterpret_cast<float*>(base + nb + nr + nx);
  a.err = c->d_err;
  HGX_CUDA(cudaFuncSetAttribute(bwm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWM_SMEM));
  HGX_CUDA(cudaFuncSetAttribute(bwm_seed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                BWM_MAX_CHUNKS * BWM_IMG_CHUNK));
  const int groups = (a.ntri + 127) / 128;
  for (int s = 0; s < p.slabs; ++s) {
    const int row0 = s * p.rows, n = std::min(p.rows, a.nrow - row0);
    if (n <= 0) break;
    bwm_item_kernel<<<dim3(p.nch, n), 256, 0, st>>>(a, row0);
    bwm_seed_kernel<<<dim3(a.ntiles, n * p.nch), 256, p.nck * BWM_IMG_CHUNK, st>>>(a, row0);
    // (the last slab may have fewer rows than ranges, the first one has at least as many)
    bwm_kernel<<<dim3(groups, std::min(p.splits, n)), BWM_THREADS, BWM_SMEM, st>>>(a, row0, n);
    HGX_CUDA(cudaGetLastError());
  }
  return HGX_OK;
}

}  // namespace hgx
