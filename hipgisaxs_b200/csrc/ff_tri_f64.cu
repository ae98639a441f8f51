// FP64 triangle form factor on detector-row grids (qz depends on the row only).
//
// The plain form (ff_tri_f64_kernel in ff_tri.cu) evaluates e^{i q.c} per q-point and triangle: a
// CUDA sincos, about 100 FP64 operations, for each of the four DWBA blocks.  Here the rotation is
// folded into the triangles (q'.c = q.(R^T c)) and e^{i q.c'} = e^{i(qx c'x + qy c'y)} e^{i qz c'z}:
// the in-plane phasor is made once per (pixel, triangle) and serves every block, the row factor
// once per (row, triangle), as in the FP32 row kernel.  Everything stays in FP64; phases are formed
// in turns, so that their reduction is exact, and the phasor is two polynomials over an eighth of
// a turn (sincos_turns).
//
// What bounds it: the FP64 pipe.  Per (pixel, triangle) with real paired blocks 40 FP64
// operations (phase 2, phasor 18, q.n~ and its products 4, sums 16).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "ff_tri_rows.cuh"
#include "turns.cuh"

namespace hgx {

constexpr int T64 = 64;         // triangles staged at a time
constexpr int F64_BLOCK = 128;

struct F64RowArgs {
  const double* sd;       // ntri x 8
  int ntri;
  const double* qx;
  const double* qy;
  const double2* rowqz;   // nrow x NK
  int nqy, nrow, ncol, rows;  // rows of a CTA
  int nsplit;
  Rot9 R;
  void* out;
  double* part;           // nsplit > 1: [split][q-point][NACC]
};

template <int U, bool PAIRED, typename OUT>
__device__ __forceinline__ void write_f64(const F64RowArgs& a, const double* T, long p) {
  constexpr int NK = PAIRED ? 4 : U;
  const int row = (int)(p / a.ncol);
  OUT* out = reinterpret_cast<OUT*>(a.out);
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
    store_ff<OUT>(out, (long)k * a.nqy + p, si / q2, -sr / q2);  // (-i) S / |q|^2
  }
}

// P pixels per thread, a thread's pixels tpr columns apart; rows x tpr threads per CTA.  The four
// double2 of a row factor of a pair hold (x, y) and (beta, gamma) (Z = x + i y, beta = qz n~z y,
// gamma = qz n~z x); a complex block's hold Z and qz n~z Z.
template <int U, bool PAIRED, int P, typename OUT>
__global__ void __launch_bounds__(F64_BLOCK, P == 2 ? 4 : 6) ff_tri_rows_f64_kernel(F64RowArgs a) {
  constexpr int NK = PAIRED ? 4 : U, NACC = PAIRED ? 8 : 2 * U;
  __shared__ double4 s_tri[T64];  // (c'x, c'y) in turns, (n~x, n~y)
  extern __shared__ __align__(16) double2 s_rf[];  // [row][triangle][unit][2]
  const int tpr = F64_BLOCK / a.rows;
  const int lr = threadIdx.x / tpr, lane = threadIdx.x - lr * tpr;
  const int row = blockIdx.y * a.rows + lr;
  const int col0 = blockIdx.x * (tpr * P) + lane;
  double qx[P], qy[P], acc[P][NACC];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int col = col0 + i * tpr;
    const bool v = row < a.nrow && col < a.ncol;
    const long p = (long)row * a.ncol + col;
    qx[i] = v ? a.qx[p] : 0.0;
    qy[i] = v ? a.qy[p] : 0.0;
#pragma unroll
    for (int n = 0; n < NACC; ++n) acc[i][n] = 0.0;
  }
  const int tiles = (a.ntri + T64 - 1) / T64;
  const int t0 = (int)((long)blockIdx.z * tiles / a.nsplit), t1 = (int)((long)(blockIdx.z + 1) * tiles / a.nsplit);
  for (int tile = t0; tile < t1; ++tile) {
    const int nt = min(T64, a.ntri - tile * T64);
    __syncthreads();
    for (int it = threadIdx.x; it < a.rows * nt; it += F64_BLOCK) {
      const int r = it / nt, j = it - r * nt, grow = blockIdx.y * a.rows + r;
      const double* t = a.sd + 8L * (tile * T64 + j);
      double np[3], cp[3];
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        np[l] = t[0] * (a.R.r[l] * t[1] + a.R.r[3 + l] * t[2] + a.R.r[6 + l] * t[3]);
        cp[l] = a.R.r[l] * t[4] + a.R.r[3 + l] * t[5] + a.R.r[6 + l] * t[6];
      }
      if (r == 0) s_tri[j] = make_double4(cp[0] * INV_TWO_PI, cp[1] * INV_TWO_PI, np[0], np[1]);
      double2* f = s_rf + (size_t)(r * T64 + j) * 2 * U;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double2 q = grow < a.nrow ? a.rowqz[(long)grow * NK + (PAIRED ? 2 * u : u)] : make_double2(0.0, 0.0);
        double s, c;
        sincos_turns(q.x * (cp[2] * INV_TWO_PI), &s, &c);
        if (PAIRED) {
          const double d = q.x * np[2];
          f[2 * u] = make_double2(c, s);
          f[2 * u + 1] = make_double2(d * s, d * c);
        } else {
          if (q.y != 0.0) {
            const double e = exp(-q.y * cp[2]);
            s *= e;
            c *= e;
          }
          const double dr = q.x * np[2], di = q.y * np[2];
          f[2 * u] = make_double2(c, s);
          f[2 * u + 1] = make_double2(dr * c - di * s, dr * s + di * c);
        }
      }
    }
    __syncthreads();
    const double2* rf = s_rf + (size_t)lr * T64 * 2 * U;
#pragma unroll 1
    for (int j = 0; j < nt; ++j, rf += 2 * U) {
      const double4 t = s_tri[j];
      double ur[P], ui[P], sn[P], cs[P];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        sincos_turns(fma(qx[i], t.x, qy[i] * t.y), &sn[i], &cs[i]);
        const double aq = fma(qx[i], t.z, qy[i] * t.w);
        ur[i] = aq * cs[i];
        ui[i] = aq * sn[i];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double2 z = rf[2 * u], d = rf[2 * u + 1];
#pragma unroll
        for (int i = 0; i < P; ++i) {
          if (PAIRED) {
            double* q = acc[i] + 4 * u % NACC;
            q[0] = fma(z.x, ur[i], fma(-d.x, sn[i], q[0]));  // P.re += x Ur - beta s
            q[1] = fma(z.x, ui[i], fma(d.x, cs[i], q[1]));   // P.im += x Ui + beta c
            q[2] = fma(-z.y, ui[i], fma(d.y, cs[i], q[2]));  // M.re += -y Ui + gamma c
            q[3] = fma(z.y, ur[i], fma(d.y, sn[i], q[3]));   // M.im += y Ur + gamma s
          } else {
            double* q = acc[i] + 2 * u % NACC;
            q[0] = fma(ur[i], z.x, fma(-ui[i], z.y, fma(d.x, cs[i], fma(-d.y, sn[i], q[0]))));
            q[1] = fma(ur[i], z.y, fma(ui[i], z.x, fma(d.x, sn[i], fma(d.y, cs[i], q[1]))));
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int col = col0 + i * tpr;
    if (row >= a.nrow || col >= a.ncol) continue;
    const long p = (long)row * a.ncol + col;
    if (a.nsplit > 1) {
      double* dst = a.part + ((size_t)blockIdx.z * a.nqy + p) * NACC;
#pragma unroll
      for (int n = 0; n < NACC; ++n) dst[n] = acc[i][n];
    } else {
      write_f64<U, PAIRED, OUT>(a, acc[i], p);
    }
  }
}

// Adds the splits' sums in a fixed order and writes the form factor.
template <int U, bool PAIRED, typename OUT>
__global__ void __launch_bounds__(F64_BLOCK) ff_tri_rows_f64_sum_kernel(F64RowArgs a) {
  constexpr int NACC = PAIRED ? 8 : 2 * U;
  const long p = (long)blockIdx.x * F64_BLOCK + threadIdx.x;
  if (p >= a.nqy) return;
  double T[NACC];
#pragma unroll
  for (int n = 0; n < NACC; ++n) T[n] = 0.0;
  for (int sp = 0; sp < a.nsplit; ++sp) {
    const double* src = a.part + ((size_t)sp * a.nqy + p) * NACC;
#pragma unroll
    for (int n = 0; n < NACC; ++n) T[n] += src[n];
  }
  write_f64<U, PAIRED, OUT>(a, T, p);
}

template <int U, bool PAIRED, int P, typename OUT>
static void launch_f64(const F64RowArgs& a, dim3 grid, cudaStream_t st) {
  ff_tri_rows_f64_kernel<U, PAIRED, P, OUT>
      <<<grid, F64_BLOCK, sizeof(double2) * 2 * U * T64 * (size_t)a.rows, st>>>(a);
}

constexpr size_t F64_PART_BYTES = (size_t)64 << 20;  // split partial sums

// Whether the row kernel (P pixels per thread, `ctas` CTAs, `nsplit` ranges of triangles) is the faster one:
// estimates per triangle in us, from 420 grids of 1 to 600 columns, 1 to 60,000 rows and 20 to 8,000 triangles.
// A CTA's time on its SM does not depend on how many of its 32 or more columns are there, so grids of few columns
// (scattered q-points count as rows of one) belong to ff_tri_f64_kernel, whose time goes with the q-points:
// 1 x 60,000 x 5,000: 4.5 against 58.8 ms, single blocks 1.5 / 49.4; 8 x 18,502 x 1,896 4.5 / 7.1.
// On the other side 16 x 24,746 x 1,253 6.9 / 6.2, 1 x 1,289 x 147 0.047 / 0.037.  Single blocks are
// taken for real (complex ones cost the plain kernel 1.5 times as much).  The margin keeps the choice within 12%
// of the plain kernel wherever it takes the row kernel.
static bool rows_f64_pays(hgx_ctx c, hgx_qgrid g, int P, long ctas, int nsplit) {
  const double sms = c->sm_count, load = (double)g->nqz / (128.0 * sms);
  const bool complex4 = g->mode == 2 && g->nk == 4;
  const double plain = complex4 ? std::max(0.295, 0.2 + 0.098 * load) : std::max(0.192, 0.13 + 0.067 * load);
  const double cta = g->nk == 1 ? (P == 1 ? 0.066 : 0.097) : complex4 ? (P == 1 ? 0.115 : 0.166) : (P == 1 ? 0.075 : 0.115);
  return !(plain < 1.15 * cta * std::max((double)ctas / sms, 1.3 / nsplit));
}

template <int U, bool PAIRED, typename OUT>
static int run_f64(hgx_ctx c, hgx_qgrid g, const double* sd, int ntri, const Rot9& R, void* out) {
  constexpr int NACC = PAIRED ? 8 : 2 * U;
  cudaStream_t st = c->stream;
  // two pixels per thread share the staged values; one where that leaves fewer CTAs than run at a
  // time, and a small image's triangles are split over CTAs too (at least two stagings each)
  const int tiles = (ntri + T64 - 1) / T64;
  int P = 2, tpr = 0;
  dim3 grid;
  for (;; --P) {
    tpr = 32;
    while (tpr < F64_BLOCK && tpr * P < g->ncol) tpr <<= 1;
    const int rows = F64_BLOCK / tpr;
    grid = dim3((g->ncol + tpr * P - 1) / (tpr * P), (g->nrow + rows - 1) / rows);
    if (P == 1 || (long)grid.x * grid.y >= 4L * c->sm_count) break;
  }
  if (grid.y > 65535u) return HGX_ERR_NO_MEMORY;  // the plain kernel takes these
  const long want = 6L * c->sm_count, ctas = (long)grid.x * grid.y;
  const size_t part = sizeof(double) * NACC * (size_t)g->nqy;
  int nsplit = (int)std::max<long>(1, std::min<long>({(want + ctas - 1) / ctas, (long)tiles / 2, 32}));
  while (nsplit > 1 && nsplit * part > F64_PART_BYTES) --nsplit;
  if (nsplit > 1 && is_capturing(st)) nsplit = 1;  // a captured call uses no workspace
  if (!rows_f64_pays(c, g, P, ctas, nsplit)) return HGX_ERR_NO_MEMORY;
  grid.z = nsplit;
  if (nsplit > 1) HGX_TRY(c->factors.reserve(nsplit * part));
  F64RowArgs a{sd, ntri, g->qx, g->qy, g->rowqz, g->nqy, g->nrow, g->ncol, F64_BLOCK / tpr, nsplit, R, out,
               reinterpret_cast<double*>(c->factors.p)};
  if (P == 2) launch_f64<U, PAIRED, 2, OUT>(a, grid, st);
  else launch_f64<U, PAIRED, 1, OUT>(a, grid, st);
  if (nsplit > 1)
    ff_tri_rows_f64_sum_kernel<U, PAIRED, OUT><<<(g->nqy + F64_BLOCK - 1) / F64_BLOCK, F64_BLOCK, 0, st>>>(a);
  HGX_CUDA(cudaGetLastError());
  return HGX_OK;
}

int ff_rows_f64(hgx_ctx c, hgx_qgrid g, const double* sd, int ntri, const Rot9& R, void* out, int ff_type) {
  const bool c64 = ff_type == HGX_C64;
  if (g->mode == 1) return c64 ? run_f64<2, true, float2>(c, g, sd, ntri, R, out) : run_f64<2, true, double2>(c, g, sd, ntri, R, out);
  if (g->nk == 4) return c64 ? run_f64<4, false, float2>(c, g, sd, ntri, R, out) : run_f64<4, false, double2>(c, g, sd, ntri, R, out);
  return c64 ? run_f64<1, false, float2>(c, g, sd, ntri, R, out) : run_f64<1, false, double2>(c, g, sd, ntri, R, out);
}

}  // namespace hgx
