// Coarse detector grids: node tables and the interpolation to pixels
// (coarse_kernels.cuh says what they are for).
#include "coarse_kernels.cuh"

#include <algorithm>
#include <cmath>

namespace spsim {

int coarse_node_count(double c, double t, double a, int digits) {
  const double cc = c > 1.0 ? c : 1.0;
  double n = 0.66 * cc + 8.9 * std::pow(cc, 0.253);
  if (t > 0.0) n += (3.5 + 11.5 * std::sqrt(cc / 320.0)) * std::pow(t, 1.2);
  if (a > 0.0) n += 6.6 * std::sqrt(a) / (1.0 + 0.5 * std::pow(cc / (8.0 * a), 0.6));
  if (digits == COARSE_DIGITS_F64) n += 10.0 + cc / 100.0;
  if (digits == COARSE_DIGITS_FULL) n += 18.0 + cc / 25.0;
  return (int)std::ceil(n);
}

CoarseAxis coarse_axis(int n_pix, double size, double centre, double distance, bool spherical) {
  CoarseAxis a;
  a.n_pix = n_pix;
  a.angular = spherical ? 0 : 1;
  a.size = size;
  a.centre = centre;
  a.distance = distance;
  a.mid = 0.0;
  a.half = 1.0;
  a.n = 0;
  a.alpha = a.asin_alpha = 0.0;
  a.to_n = 0;
  a.to_alpha = a.to_asin = 0.0;
  a.derivative = 0;
  if (a.angular) {
    const double edge = 0.5 * (n_pix - 1) / n_pix * size;
    const double t0 = std::atan((-edge - centre) / distance), t1 = std::atan((edge - centre) / distance);
    a.mid = 0.5 * (t0 + t1);
    a.half = 0.5 * (t1 - t0);
  }
  return a;
}

// The stretch leaves errors of e^-(n acosh(1 / alpha)) whatever the function:
// e^-(9.3 n^(1/3)) is small enough for 1e-8 at eight nodes and for 1e-12 at the
// twenty that these take; for 1e-15 e^-36 at least.
void coarse_set_nodes(CoarseAxis &a, int n, int digits) {
  a.n = n;
  double stretch = 9.3 * std::cbrt((double)n);
  if (digits == COARSE_DIGITS_FULL) stretch = std::max(stretch, 36.0);
  a.alpha = 1.0 / std::cosh(stretch / n);
  a.asin_alpha = std::asin(a.alpha);
}

// ---------------------------------------------------------------------------
// node q vectors and interpolation matrices

struct CoarseTables {
  DetGeom g;
  CoarseAxis x, y;
  int ldx, ldy, ltx, lty;
  double *q64, *mx, *my, *tx, *ty;
};

// position on the detector (m) of node k of an axis
__device__ __forceinline__ double coarse_node_pos(const CoarseAxis &a, int k) {
  const double X = asin(a.alpha * cospi((double)k / (a.n - 1))) / a.asin_alpha;
  if (a.angular) return a.distance * tan(a.mid + a.half * X);
  return (0.5 * (a.n_pix - 1) * X / a.n_pix) * a.size - a.centre;
}

// points interpolated to
__host__ __device__ __forceinline__ int coarse_rows(const CoarseAxis &a) { return a.to_n > 0 ? a.to_n : a.n_pix; }

// Where column k of a matrix row is stored: of each eight, k and k + 4 are
// neighbours, a lane's pair in dmma_tile.
__device__ __forceinline__ int coarse_slot(int k) { return (k & ~7) | (2 * (k & 3) + ((k >> 2) & 1)); }

// One row (point p) of an interpolation matrix by one warp:
// M[k] = (w_k / (xi - xi_k)) / sum_j w_j / (xi - xi_j), the barycentric weights
// of the Chebyshev extreme points w_k = (-1)^k, halved at both ends.
// mt: the transpose, [node][lt], or nullptr.
__device__ __forceinline__ void coarse_row(int p, const CoarseAxis &a, int ld, double *__restrict__ m, int lt,
                                           double *__restrict__ mt) {
  const int lane = threadIdx.x & 31, n = a.n;
  double X = 2.0 * p / (a.n_pix - 1) - 1.0;
  if (a.to_n > 0) {
    X = asin(a.to_alpha * cospi((double)p / (a.to_n - 1))) / a.to_asin;
  } else if (a.angular) {
    const double pos = ((p - (a.n_pix - 1.0) / 2.0) / a.n_pix) * a.size - a.centre;
    X = (atan(pos / a.distance) - a.mid) / a.half;
  }
  if (a.derivative) {
    // by a central difference: its own error is 1e-6 of the derivative at most
    // (step 1e-5 of the half axis, 1,024 nodes)
    const double step = 1e-5;
    const double x1 = sin(a.asin_alpha * (X + step)) / a.alpha, x0 = sin(a.asin_alpha * (X - step)) / a.alpha;
    double s1 = 0.0, s0 = 0.0;
    for (int pass = 0; pass < 2; ++pass) {
      for (int k = lane; k < (pass ? ld : n); k += 32) {
        const double node = cospi((double)k / (n - 1));
        const double w = ((k & 1) ? -1.0 : 1.0) * ((k == 0 || k == n - 1) ? 0.5 : 1.0);
        // a node within 1e-14 of a stepped point counts as 1e-14 away
        const double d1 = copysign(fmax(fabs(x1 - node), 1e-14), x1 - node);
        const double d0 = copysign(fmax(fabs(x0 - node), 1e-14), x0 - node);
        if (!pass) {
          s1 += w / d1;
          s0 += w / d0;
        } else {
          m[(long long)p * ld + coarse_slot(k)] = k < n ? (w / d1 / s1 - w / d0 / s0) / (2.0 * step) : 0.0;
        }
      }
      if (!pass)
        for (int o = 16; o > 0; o >>= 1) {
          s1 += __shfl_xor_sync(0xffffffffu, s1, o);
          s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        }
    }
    return;
  }
  const double xi = sin(a.asin_alpha * X) / a.alpha;
  double sum = 0.0;
  int hit = -1;
  for (int k = lane; k < n; k += 32) {
    const double d = xi - cospi((double)k / (n - 1));
    if (fabs(d) < 1e-14) hit = k;
    const double w = ((k & 1) ? -1.0 : 1.0) * ((k == 0 || k == n - 1) ? 0.5 : 1.0);
    sum += hit == k ? 0.0 : w / d;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    hit = max(hit, __shfl_xor_sync(0xffffffffu, hit, o));
  }
  for (int k = lane; k < ld; k += 32) {
    double v = 0.0;
    if (k < n) {
      const double d = xi - cospi((double)k / (n - 1));
      const double w = ((k & 1) ? -1.0 : 1.0) * ((k == 0 || k == n - 1) ? 0.5 : 1.0);
      v = hit >= 0 ? (k == hit ? 1.0 : 0.0) : w / d / sum;
    }
    m[(long long)p * ld + coarse_slot(k)] = v;
    if (mt && k < n) {
      mt[(long long)k * lt + coarse_slot(p)] = v;
      if (p == coarse_rows(a) - 1)
        for (int z = p + 1; z < lt; ++z) mt[(long long)k * lt + coarse_slot(z)] = 0.0;
    }
  }
}

__global__ void __launch_bounds__(256) coarse_tables_kernel(CoarseTables t) {
  const int warp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const int nx = coarse_rows(t.x), ny = coarse_rows(t.y);
  if (warp < nx) {
    coarse_row(warp, t.x, t.ldx, t.mx, t.ltx, t.tx);
  } else if (warp < nx + ny) {
    coarse_row(warp - nx, t.y, t.ldy, t.my, t.lty, t.ty);
  } else {
    const int i = (warp - nx - ny) * 32 + lane;
    if (i >= t.x.n * t.y.n) return;
    const double px = coarse_node_pos(t.x, i % t.x.n), py = coarse_node_pos(t.y, i / t.x.n);
    double q0, q1, q2 = 0.0;
    if (t.g.spherical) {
      q0 = t.g.fpx * px / t.g.px_size;
      q1 = t.g.fpy * py / t.g.py_size;
    } else {
      const double r = sqrt(px * px + py * py + t.g.distance * t.g.distance);
      q0 = px / r * t.g.ewald;
      q1 = py / r * t.g.ewald;
      q2 = (t.g.distance / r - 1.0) * t.g.ewald;
    }
    q2 += t.g.lift;
    t.q64[3 * i] = q0;
    t.q64[3 * i + 1] = q1;
    t.q64[3 * i + 2] = q2;
  }
}

cudaError_t launch_coarse_tables(const DetGeom &g, const CoarseAxis &x, const CoarseAxis &y, double *q64, double *mx,
                                 double *my, cudaStream_t st, double *tx, double *ty) {
  CoarseTables t;
  t.g = g;
  t.x = x;
  t.y = y;
  t.ldx = coarse_ld(x.n);
  t.ldy = coarse_ld(y.n);
  t.q64 = q64;
  t.mx = mx;
  t.my = my;
  t.ltx = coarse_ld(x.n_pix);
  t.lty = coarse_ld(y.n_pix);
  t.tx = tx;
  t.ty = ty;
  const long long warps = (long long)coarse_rows(x) + coarse_rows(y) + ((long long)x.n * y.n + 31) / 32;
  coarse_tables_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(t);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Interpolation as two FP64 matrix products on the tensor pipe (m8n8k4):
//   columns  strip[k][x] = sum_i M_x[x][i] nodes[k][i]
//   rows     pixel[y][x] = sum_k M_y[y][k] strip[k][x]
// The rows' kernel then applies the global B factor and the centre phase and writes F
// and |F|^2 as sf_finalize_kernel does.  Fragments come straight from L1 / L2:
// a warp's RM x RN tiles of 8 x 8 complex values take RM + 2 RN 16-byte loads
// per eight k.  FP64 MMA runs at the FMA units' own rate but issues a quarter of
// the loads of the same product written with FMAs from shared memory (1024^2
// pixels from 182 nodes a side: that form took 335 us, both products now 58).
constexpr int INTERP_WARPS_M = 2, INTERP_WARPS_N = 2;
constexpr int INTERP_THREADS = 32 * INTERP_WARPS_M * INTERP_WARPS_N;

__device__ __forceinline__ void dmma(double c[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// M B by one warp for RM x RN tiles of 8 x 8 complex values: M's rows from m0
// (in range, clamped), B's column n0 + 8 j + fr from bcol[j], bstep values from
// one k to the next.  A tile's real and imaginary parts are two MMA tiles, so
// that a lane reads a complex value at a time.  Of each group of eight k the
// lane's entries are k = fc + 4 s in step s: neighbours in M (coarse_slot), and
// of B's rows four lanes read 64 bytes (with k = 2 fc + s every other 16: the
// columns of 65 cells 20 us instead of 15).  M holds zeros from k_all to its
// padded end, where B is read at its last row.
// AHEAD: the groups whose fragments are read ahead of the one multiplied (L2's
// latency bounds the small tiles, registers the large ones).
template <int RM, int RN, int AHEAD>
__device__ __forceinline__ void dmma_tile(const double *__restrict__ M, int ld, int m0, int m_all,
                                          const double2 *const bcol[RN], long long bstep, int k_all, int k_first,
                                          int k_end, double re[RM][RN][2], double im[RM][RN][2]) {
  const int lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
  const double2 *arow[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) arow[i] = (const double2 *)(M + (long long)min(m0 + 8 * i + fr, m_all - 1) * ld) + fc;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  double2 a[AHEAD + 1][RM], b0[AHEAD + 1][RN], b1[AHEAD + 1][RN];
  auto load = [&](int k, int slot) {
    const long long kb0 = min(k + fc, k_all - 1) * bstep, kb1 = min(k + fc + 4, k_all - 1) * bstep;
#pragma unroll
    for (int i = 0; i < RM; ++i) a[slot][i] = arow[i][k / 2];
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      b0[slot][j] = bcol[j][kb0];
      b1[slot][j] = bcol[j][kb1];
    }
  };
#pragma unroll
  for (int s = 0; s < AHEAD; ++s)
    if (k_first + 8 * s < k_end) load(k_first + 8 * s, s);
  for (int k0 = k_first; k0 < k_end; k0 += 8 * (AHEAD + 1)) {
#pragma unroll
    for (int s = 0; s <= AHEAD; ++s) {
      const int k = k0 + 8 * s;
      if (k >= k_end) break;
      if (k + 8 * AHEAD < k_end) load(k + 8 * AHEAD, (s + AHEAD) % (AHEAD + 1));
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          dmma(re[i][j], a[s][i].x, b0[s][j].x);
          dmma(im[i][j], a[s][i].x, b0[s][j].y);
        }
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          dmma(re[i][j], a[s][i].y, b1[s][j].x);
          dmma(im[i][j], a[s][i].y, b1[s][j].y);
        }
    }
  }
}

// ROWS: the second product, else the first.  SUM: of a cell (CoarsePattern::sum).
// BOTH: the second product after the first one's for the block's own 16 columns,
// in shared memory, on grids of up to 64 x 64 nodes.
constexpr int BOTH_NODES = 64;
template <int RM, int RN, int AHEAD, bool ROWS, bool SUM, bool BOTH>
__global__ void __launch_bounds__(INTERP_THREADS, 7)
    coarse_interp_kernel(const __grid_constant__ CoarseBatch batch, int pattern0, double2 *__restrict__ strips,
                         long long strip_stride) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pattern = pattern0 + blockIdx.z;
  CoarsePattern cp = batch.pats ? batch.coarse[pattern] : batch.one;
  if (!batch.pats) cp.nodes += (long long)pattern * cp.nyn * cp.nxn;
  double2 *__restrict__ strip = strips + blockIdx.z * strip_stride;
  const int m_all = ROWS ? cp.ny : cp.nx;             // rows of the left matrix
  const int n_all = ROWS ? cp.nx : cp.nyn;            // columns of the right one
  const int k_all = ROWS ? cp.nyn : cp.nxn;
  const int ld = ROWS ? cp.ldy : cp.ldx;
  const double *__restrict__ M = ROWS ? cp.my : cp.mx;
  const int m0 = (blockIdx.y * INTERP_WARPS_M + warp % INTERP_WARPS_M) * (8 * RM);
  const int n0 = (blockIdx.x * INTERP_WARPS_N + warp / INTERP_WARPS_M) * (8 * RN);
  const int fr = lane >> 2, fc = lane & 3;
  constexpr int CLD = 17;
  __shared__ double2 columns[BOTH ? BOTH_NODES * CLD : 1];
  if (BOTH) {
    static_assert(!BOTH || (RN == 1 && INTERP_WARPS_N == 2), "16 columns per block");
    const int x0 = blockIdx.x * 16 + 8 * (warp & 1);
    for (int kb = 16 * (warp >> 1); kb < cp.nyn; kb += 32) {
      const double2 *col[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) col[j] = cp.nodes + (long long)min(kb + 8 * j + fr, cp.nyn - 1) * cp.nxn;
      double cr[1][2][2], ci[1][2][2];
      dmma_tile<1, 2, 2>(cp.mx, cp.ldx, x0, cp.nx, col, 1, cp.nxn, 0, cp.nxn, cr, ci);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        columns[(kb + 8 * (j >> 1) + 2 * fc + (j & 1)) * CLD + 8 * (warp & 1) + fr] =
            make_double2(cr[0][j >> 1][j & 1], ci[0][j >> 1][j & 1]);
    }
    __syncthreads();
  }
  if (m0 >= m_all || n0 >= n_all) return;

  const double2 *bcol[RN];
#pragma unroll
  for (int j = 0; j < RN; ++j) {
    const int n = min(n0 + 8 * j + fr, n_all - 1);
    bcol[j] = BOTH   ? columns + (n0 - (int)blockIdx.x * 16 + 8 * j + fr)
              : ROWS ? strip + n
                     : cp.nodes + (long long)n * cp.nxn;
  }
  double re_[RM][RN][2], im_[RM][RN][2];
  dmma_tile<RM, RN, AHEAD>(M, ld, m0, m_all, bcol, BOTH ? CLD : ROWS ? cp.nx : 1, k_all, 0, k_all, re_, im_);

  if (!ROWS) {
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int x = m0 + 8 * i + fr;
      if (x >= cp.nx) continue;
#pragma unroll
      for (int j = 0; j < 2 * RN; ++j) {
        const int k = n0 + 8 * (j >> 1) + 2 * fc + (j & 1);
        if (k < cp.nyn) strip[(long long)k * cp.nx + x] = make_double2(re_[i][j >> 1][j & 1], im_[i][j >> 1][j & 1]);
      }
    }
    return;
  }
  const long long npix = (long long)cp.nx * cp.ny;
  const double *q64 = batch.q64, *rot = batch.rots ? batch.rots + 9LL * pattern : nullptr, *center = batch.center;
  double qscale = 1.0;
  float2 *F = batch.F ? batch.F + pattern * npix : nullptr;
  float *I = batch.I ? batch.I + pattern * npix : nullptr;
  if (batch.pats) {
    const SfPattern &pt = batch.pats[cp.parent];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && pt.mol_err && *pt.mol_err) atomicOr(pt.plan_err, 1);
    q64 = pt.q64;
    rot = pt.has_rot ? pt.rot : nullptr;
    center = SUM ? cp.shift : pt.center;
    qscale = pt.qscale;
    F = pt.F;
    I = pt.I;
  }
  // the tile by rows of neighbouring pixels, one per lane: coalesced, and the
  // phase's code once instead of once per accumulator
  constexpr int TN = 8 * RN, TLD = TN + 1;
  __shared__ double2 tiles[INTERP_WARPS_M * INTERP_WARPS_N][8 * RM * TLD];
  double2 *tile = tiles[warp];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 2 * RN; ++j)
      tile[(8 * i + fr) * TLD + 8 * (j >> 1) + 2 * fc + (j & 1)] =
          make_double2(re_[i][j >> 1][j & 1], im_[i][j >> 1][j & 1]);
  __syncwarp();
  const bool need_q = SUM || F || cp.B != 0.0;
#pragma unroll 1
  for (int e = lane; e < 8 * RM * TN; e += 32) {
    const int y = m0 + e / TN, x = n0 + e % TN;
    if (y >= cp.ny || x >= cp.nx) continue;
    const long long p = (long long)y * cp.nx + x;
    const double2 v = tile[e / TN * TLD + e % TN];
    double re = v.x, im = v.y;
    if (need_q) {
      const double a = q64[3 * p], b = q64[3 * p + 1], c = q64[3 * p + 2];
      if (!SUM && cp.B != 0.0) {
        const double w = exp(-cp.B * 0.25e-20 * (a * a + b * b + c * c));
        re *= w;
        im *= w;
      }
      if (SUM || F) {
        double ux = a, uy = b, uz = c;
        if (rot) {
          ux = rot[0] * a + rot[1] * b + rot[2] * c;
          uy = rot[3] * a + rot[4] * b + rot[5] * c;
          uz = rot[6] * a + rot[7] * b + rot[8] * c;
        }
        double t = (ux * center[0] + uy * center[1] + uz * center[2]) * qscale;
        t -= rint(t);
        double sn, cs;
        sincospi(2.0 * t, &sn, &cs);
        if (SUM) {
          atomicAdd(&cp.sum[p].x, re * cs + im * sn);
          atomicAdd(&cp.sum[p].y, im * cs - re * sn);
          continue;
        }
        F[p] = make_float2((float)(re * cs + im * sn), (float)(im * cs - re * sn));
      }
    }
    if (cp.out)
      cp.out[p] = make_double2(re, im);
    else if (I)
      I[p] = (float)(re * re + im * im);
  }
}

// The second product of many cells: as above onto the pattern's own nodes,
// per_block cells in turn by one block, which adds them up in shared memory with
// the phases of their centres and goes to the pattern's sums once per pattern.
// 128 x 65 cells to 38^2 nodes: one cell per block, each adding to the sums,
// 191 us, which the atomics bound; 133 us with nine, 153 with sixteen.  Where a
// block takes one cell, the other kernel (65 cells to 167^2 nodes: 47 us, 62 here).
__global__ void __launch_bounds__(INTERP_THREADS, 6)
    cell_rows_kernel(const __grid_constant__ CoarseBatch batch, int cell0, int n, int per_block,
                     const double2 *__restrict__ strips, long long strip_stride) {
  constexpr int RM = 2, RN = 1, TN = 8 * RN, TLD = TN + 1, POINTS = 8 * RM * TN;
  __shared__ double2 tiles[INTERP_WARPS_M * INTERP_WARPS_N][8 * RM * TLD];
  __shared__ double2 sums[INTERP_WARPS_M * INTERP_WARPS_N][POINTS];
  __shared__ double us[INTERP_WARPS_M * INTERP_WARPS_N][3][POINTS];  // R q of the warp's nodes
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
  const int m0 = (blockIdx.y * INTERP_WARPS_M + warp % INTERP_WARPS_M) * (8 * RM);
  const int n0 = (blockIdx.x * INTERP_WARPS_N + warp / INTERP_WARPS_M) * (8 * RN);
  double2 *tile = tiles[warp], *sum = sums[warp];
  double(*u)[POINTS] = us[warp];
  double2 *to = nullptr;
  int to_nx = 0, to_ny = 0;
  auto flush = [&]() {
    for (int e = lane; e < POINTS && to; e += 32) {
      const int y = m0 + e / TN, x = n0 + e % TN;
      if (y >= to_ny || x >= to_nx) continue;
      atomicAdd(&to[(long long)y * to_nx + x].x, sum[e].x);
      atomicAdd(&to[(long long)y * to_nx + x].y, sum[e].y);
    }
  };
  double qscale = 1.0;
  const int first = blockIdx.z * per_block, end = min(first + per_block, n);
  for (int c = first; c < end; ++c) {
    const CoarsePattern &cp = batch.coarse[cell0 + c];
    if (cp.sum != to) {
      flush();
      to = cp.sum;
      to_nx = cp.nx;
      to_ny = cp.ny;
      const SfPattern &pt = batch.pats[cp.parent];
      qscale = pt.qscale;
      for (int e = lane; e < POINTS; e += 32) {
        const int y = m0 + e / TN, x = n0 + e % TN;
        sum[e] = make_double2(0.0, 0.0);
        if (y >= to_ny || x >= to_nx) continue;
        const double *q = pt.q64 + 3 * ((long long)y * to_nx + x), *R = pt.rot;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          u[k][e] = pt.has_rot ? R[3 * k] * q[0] + R[3 * k + 1] * q[1] + R[3 * k + 2] * q[2] : q[k];
      }
    }
    if (m0 >= to_ny || n0 >= to_nx) continue;
    const double2 *bcol[RN] = {strips + c * strip_stride + min(n0 + fr, to_nx - 1)};
    double re[RM][RN][2], im[RM][RN][2];
    dmma_tile<RM, RN, 1>(cp.my, cp.ldy, m0, to_ny, bcol, to_nx, cp.nyn, 0, cp.nyn, re, im);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) tile[(8 * i + fr) * TLD + 2 * fc + h] = make_double2(re[i][0][h], im[i][0][h]);
    __syncwarp();
#pragma unroll 2
    for (int e = lane; e < POINTS; e += 32) {
      const int y = m0 + e / TN, x = n0 + e % TN;
      if (y >= to_ny || x >= to_nx) continue;
      double t = (u[0][e] * cp.shift[0] + u[1][e] * cp.shift[1] + u[2][e] * cp.shift[2]) * qscale;
      t -= rint(t);
      double sn, cs;
      sincospi(2.0 * t, &sn, &cs);
      const double2 v = tile[e / TN * TLD + e % TN];
      sum[e].x += v.x * cs + v.y * sn;
      sum[e].y += v.y * cs - v.x * sn;
    }
  }
  flush();
}

template <int RM, int RN, int AHEAD, bool ROWS, bool SUM = false, bool BOTH = false>
static void interp_t(const CoarseBatch &b, int pattern0, int n, int m_max, int n_max, double2 *strip, long long stride,
                     cudaStream_t st) {
  const int bm = 8 * RM * INTERP_WARPS_M, bn = 8 * RN * INTERP_WARPS_N;
  dim3 grid((unsigned)((n_max + bn - 1) / bn), (unsigned)((m_max + bm - 1) / bm), (unsigned)n);
  coarse_interp_kernel<RM, RN, AHEAD, ROWS, SUM, BOTH><<<grid, INTERP_THREADS, 0, st>>>(b, pattern0, strip, stride);
}

cudaError_t launch_coarse_interp(const CoarseBatch &b, int npat, int max_nx, int max_ny, int max_nxn, int max_nyn,
                                 double2 *strip, long long strip_size, cudaStream_t st, bool cells) {
  if (npat <= 0 || max_nx <= 0 || max_ny <= 0) return cudaSuccess;
  const long long stride = (long long)max_nyn * max_nx;
  const int group = (int)std::min<long long>(std::max<long long>(strip_size / stride, 1), 65535);
  for (int p0 = 0; p0 < npat; p0 += group) {
    const int n = std::min(group, npat - p0);
    // Columns: 8 x 8 values per warp (50,000 atoms x 1024^2, 161 nodes a side:
    // 10.4 us, with 16 x 8 11.8, 16 x 16 14).  Rows: 16 x 8 (44 us; 8 x 8 64,
    // 32 x 16 46.5), but 8 x 8 where those leave most SMs without two blocks
    // (one 512^2 pattern: 6.4 us instead of 8.8; eight: 43 instead of 34).
    const long long tiles = (long long)((max_ny + 31) / 32) * ((max_nx + 15) / 16);
    // Both products in one launch where the second leaves SMs without two blocks
    // and the first is short: one 256^2 pattern 7.3 us instead of 3.3 + 6.0 and a
    // launch (the call 16.4 us instead of 20.5).  Not beyond: 517 x 389 pixels from
    // 54 x 45 nodes 21 us against 5 + 11, eight 512^2 patterns 53 against 4 + 33.
    if (!cells && max_nxn <= BOTH_NODES && max_nyn <= BOTH_NODES && n * tiles < 2 * 148) {
      interp_t<1, 1, 2, true, false, true>(b, p0, n, max_ny, max_nx, strip, stride, st);
      continue;
    }
    interp_t<1, 1, 2, false>(b, p0, n, max_nx, max_nyn, strip, stride, st);
    // cells: as many per block as leave each SM's six blocks six turns
    const int per_block = (int)std::min<long long>(n * tiles / (36 * 148), 16);
    if (cells && per_block <= 1) {
      interp_t<2, 1, 1, true, true>(b, p0, n, max_ny, max_nx, strip, stride, st);
    } else if (cells) {
      dim3 grid((unsigned)((max_nx + 15) / 16), (unsigned)((max_ny + 31) / 32),
                (unsigned)((n + per_block - 1) / per_block));
      cell_rows_kernel<<<grid, INTERP_THREADS, 0, st>>>(b, p0, n, per_block, strip, stride);
    } else if (n * tiles < 2 * 148) {
      interp_t<1, 1, 2, true>(b, p0, n, max_ny, max_nx, strip, stride, st);
    } else {
      interp_t<2, 1, 1, true>(b, p0, n, max_ny, max_nx, strip, stride, st);
    }
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// the adjoint of the interpolation: H_nodes = M_y^T H M_x with
// H = dL/d|F|^2 A e^{-B s^2} per pixel, A the centred amplitude

__global__ void __launch_bounds__(256)
    coarse_adjoint_pixels_kernel(CoarseAdjoint a, int pattern0, double2 *__restrict__ H) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.npix) return;
  const int pat = pattern0 + blockIdx.y;
  const double q0 = a.q64[3 * p], q1 = a.q64[3 * p + 1], q2 = a.q64[3 * p + 2];
  double ux = q0, uy = q1, uz = q2;
  if (a.rot) {
    const double *R = a.rot + 9LL * pat;
    ux = R[0] * q0 + R[1] * q1 + R[2] * q2;
    uy = R[3] * q0 + R[4] * q1 + R[5] * q2;
    uz = R[6] * q0 + R[7] * q1 + R[8] * q2;
  }
  double t = ux * a.center[0] + uy * a.center[1] + uz * a.center[2];
  t -= rint(t);
  double sn, cs;
  sincospi(2.0 * t, &sn, &cs);
  const float2 F = a.F[pat * a.npix + p];
  double h = a.G[pat * a.npix + p];
  if (a.B != 0.0) h *= exp(-a.B * 0.25e-20 * (q0 * q0 + q1 * q1 + q2 * q2));
  H[blockIdx.y * a.npix + p] = make_double2(h * (F.x * cs - F.y * sn), h * (F.x * sn + F.y * cs));
}

// out[m][n] = sum_k L[m][k] R[n][k] for complex R of n_all rows, k_all long, and
// real L of m_all rows, ld long; blockIdx.z: pattern.  Few results of long sums
// (30 nodes a side, k a side of the detector): one 8 x 8 tile per block, its
// warps taking a quarter of k each, their parts added in a fixed order.  Eight
// 512^2 patterns (k = 512 both times): 16.5 and 6.5 us; 45 and 44 us with 16 x 16
// tiles of all of k per warp, 18 and 14 with 8 x 8 tiles of all of k.
constexpr int PRODUCT_SPLIT = 4;
__global__ void __launch_bounds__(32 * PRODUCT_SPLIT)
    coarse_product_kernel(const double *__restrict__ L, int ld, int m_all, const double2 *__restrict__ R, int n_all,
                          int k_all, double2 *__restrict__ out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
  const int m0 = blockIdx.y * 8, n0 = blockIdx.x * 8;
  R += (long long)blockIdx.z * n_all * k_all;
  out += (long long)blockIdx.z * m_all * n_all;
  const double2 *bcol[1] = {R + (long long)min(n0 + fr, n_all - 1) * k_all};
  const int part = (k_all + 8 * PRODUCT_SPLIT - 1) / (8 * PRODUCT_SPLIT) * 8;
  double re[1][1][2], im[1][1][2];
  dmma_tile<1, 1, 3>(L, ld, m0, m_all, bcol, 1, k_all, warp * part, min((warp + 1) * part, k_all), re, im);
  __shared__ double2 parts[PRODUCT_SPLIT][64];
#pragma unroll
  for (int h = 0; h < 2; ++h) parts[warp][8 * fr + 2 * fc + h] = make_double2(re[0][0][h], im[0][0][h]);
  __syncthreads();
  const int m = m0 + threadIdx.x / 8, n = n0 + threadIdx.x % 8;
  if (threadIdx.x >= 64 || m >= m_all || n >= n_all) return;
  double2 v = parts[0][threadIdx.x];
#pragma unroll
  for (int w = 1; w < PRODUCT_SPLIT; ++w) {
    v.x += parts[w][threadIdx.x].x;
    v.y += parts[w][threadIdx.x].y;
  }
  out[(long long)m * n_all + n] = v;
}

static void product(const double *L, int ld, int m, const double2 *R, int n, int k, double2 *out, int npat,
                    cudaStream_t st) {
  dim3 grid((unsigned)((n + 7) / 8), (unsigned)((m + 7) / 8), (unsigned)npat);
  coarse_product_kernel<<<grid, 32 * PRODUCT_SPLIT, 0, st>>>(L, ld, m, R, n, k, out);
}

cudaError_t launch_coarse_adjoint(const CoarseAdjoint &a, int npat, double2 *H, int group, double2 *strip,
                                  double2 *nodes, cudaStream_t st) {
  for (int p0 = 0; p0 < npat; p0 += group) {
    const int n = std::min(group, npat - p0);
    dim3 grid((unsigned)((a.npix + 255) / 256), (unsigned)n);
    coarse_adjoint_pixels_kernel<<<grid, 256, 0, st>>>(a, p0, H);
    // strip[i][y] = sum_x M_x[x][i] H[y][x], then nodes[k][i] = sum_y M_y[y][k] strip[i][y]
    product(a.tx, coarse_ld(a.nx), a.nxn, H, a.ny, a.nx, strip, n, st);
    product(a.ty, coarse_ld(a.ny), a.nyn, strip, a.nxn, a.ny, nodes + (long long)p0 * a.nyn * a.nxn, n, st);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// patterns on a detector's rounded HKL list

// Bound by its FP64 arithmetic and 64 bytes of amplitudes per pixel.
__global__ void __launch_bounds__(256) list_combine_kernel(const __grid_constant__ ListCombine c, long long p0,
                                                           long long p1) {
  const long long p = p0 + (long long)blockIdx.x * 256 + threadIdx.x;
  if (p >= p1) return;
  const DetGeom &g = c.g;
  const int x = (int)(p % g.nx), y = (int)(p / g.nx);
  const double px = ((x - (g.nx - 1.0) / 2.0) / g.nx) * g.width - g.cx;
  const double py = ((y - (g.ny - 1.0) / 2.0) / g.ny) * g.height - g.cy;
  // q of the detector and its derivatives by X and Y
  double q[3], gx[3], gy[3];
  if (g.spherical) {
    const double hx = 0.5 * (g.nx - 1) / g.nx * g.width, hy = 0.5 * (g.ny - 1) / g.ny * g.height;
    q[0] = g.fpx * px / g.px_size;
    q[1] = g.fpy * py / g.py_size;
    q[2] = 0.0;
    gx[0] = g.fpx * hx / g.px_size;
    gy[1] = g.fpy * hy / g.py_size;
    gx[1] = gx[2] = gy[0] = gy[2] = 0.0;
  } else {
    const double d = g.distance, ir = rsqrt(px * px + py * py + d * d), ir2 = ir * ir;
    const double v[3] = {px, py, d};
    const double dx = c.x.half * (d + px * px / d) * ir * g.ewald, dy = c.y.half * (d + py * py / d) * ir * g.ewald;
    for (int k = 0; k < 3; ++k) {
      q[k] = v[k] * ir * g.ewald - (k == 2 ? g.ewald : 0.0);
      gx[k] = ((k == 0 ? 1.0 : 0.0) - v[k] * px * ir2) * dx;
      gy[k] = ((k == 1 ? 1.0 : 0.0) - v[k] * py * ir2) * dy;
    }
  }
  const double l[3] = {c.hkl[3 * p], c.hkl[3 * p + 1], c.hkl[3 * p + 2]};
  double e[3], d[3];  // the list's difference, in its frame and in the detector's
  for (int k = 0; k < 3; ++k) e[k] = l[k] - (c.rot[3 * k] * q[0] + c.rot[3 * k + 1] * q[1] + c.rot[3 * k + 2] * q[2]);
  for (int k = 0; k < 3; ++k) d[k] = c.rot[k] * e[0] + c.rot[3 + k] * e[1] + c.rot[6 + k] * e[2];
  const double det = 1.0 / (gx[0] * gy[1] - gx[1] * gy[0]);
  const double u = (d[0] * gy[1] - d[1] * gy[0]) * det, v = (gx[0] * d[1] - gx[1] * d[0]) * det;
  const double w = (d[2] - u * gx[2] - v * gy[2]) / c.lift;
  const double2 a = c.a[p], ax = c.ax[p], ay = c.ay[p], b = c.lifted[p];
  double re = a.x + u * ax.x + v * ay.x + w * (b.x - a.x);
  double im = a.y + u * ax.y + v * ay.y + w * (b.y - a.y);
  if (c.B != 0.0) {
    const double f = exp(-c.B * 0.25e-20 * (l[0] * l[0] + l[1] * l[1] + l[2] * l[2]));
    re *= f;
    im *= f;
  }
  if (c.I) c.I[p] = (float)(re * re + im * im);
  if (c.F) {
    double t = l[0] * c.center[0] + l[1] * c.center[1] + l[2] * c.center[2];
    t -= rint(t);
    double sn, cs;
    sincospi(2.0 * t, &sn, &cs);
    c.F[p] = make_float2((float)(re * cs + im * sn), (float)(im * cs - re * sn));
  }
}

cudaError_t launch_list_combine(const ListCombine &c, long long p0, long long p1, cudaStream_t st) {
  if (p1 <= p0) return cudaSuccess;
  list_combine_kernel<<<(unsigned)((p1 - p0 + 255) / 256), 256, 0, st>>>(c, p0, p1);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// atoms by cells

__device__ __forceinline__ double cell_centre(const CellLattice &l, int i, int sub) {
  return l.a * (i - l.reach + 0.5 * sub);
}

__global__ void __launch_bounds__(TILE_ATOMS)
    cells_count_kernel(CellLattice l, const AtomD *__restrict__ atoms, const int *__restrict__ perm,
                       const TileDesc *__restrict__ tiles, int n_elem, int *__restrict__ key, int *__restrict__ count) {
  const TileDesc t = tiles[blockIdx.x];
  if ((int)threadIdx.x >= t.count) return;
  const int i = t.atom_begin + threadIdx.x;
  if (perm[i] < 0) return;
  const double r[3] = {atoms[i].x, atoms[i].y, atoms[i].z};
  int at[2][3];
  double d[2] = {0.0, 0.0};
#pragma unroll
  for (int sub = 0; sub < 2; ++sub)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      at[sub][k] = min(max((int)rint(r[k] / l.a - 0.5 * sub) + l.reach, 0), l.dim - 1);
      const double e = r[k] - cell_centre(l, at[sub][k], sub);
      d[sub] += e * e;
    }
  const int sub = d[1] < d[0];
  const int cell = ((sub * l.dim + at[sub][2]) * l.dim + at[sub][1]) * l.dim + at[sub][0];
  key[i] = cell * n_elem + t.elem;
  atomicAdd(&count[cell * n_elem + t.elem], 1);
}

__global__ void __launch_bounds__(256)
    cells_order_kernel(const int *__restrict__ perm, int n_padded, const int *__restrict__ key,
                       const int *__restrict__ run_begin, int *__restrict__ cursor, int *__restrict__ order) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_padded || perm[i] < 0) return;
  order[run_begin[key[i]] + atomicAdd(&cursor[key[i]], 1)] = i;
}

// each atom's place in its run by counting those before it, so that the sums'
// order does not depend on the atomics'
__global__ void __launch_bounds__(256)
    cells_place_kernel(CellLattice l, const AtomD *__restrict__ atoms, const int *__restrict__ perm, int n_padded,
                       int n_elem, const int *__restrict__ key, const int *__restrict__ count,
                       const int *__restrict__ run_begin, const int *__restrict__ order, AtomD *__restrict__ out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_padded || perm[i] < 0) return;
  const int k = key[i], begin = run_begin[k], n = count[k];
  int rank = 0;
#pragma unroll 8
  for (int s = 0; s < n; ++s) rank += order[begin + s] < i;
  const int cell = k / n_elem;
  const int x = cell % l.dim, y = cell / l.dim % l.dim, z = cell / (l.dim * l.dim) % l.dim;
  const int sub = cell / (l.dim * l.dim * l.dim);
  AtomD a = atoms[i];
  a.x -= cell_centre(l, x, sub);
  a.y -= cell_centre(l, y, sub);
  a.z -= cell_centre(l, z, sub);
  out[begin + rank] = a;
}

cudaError_t launch_cells_count(const CellLattice &l, const AtomD *atoms, const int *perm, const TileDesc *tiles,
                               int n_tiles, int n_elem, int *key, int *count, cudaStream_t st) {
  if (n_tiles > 0) cells_count_kernel<<<n_tiles, TILE_ATOMS, 0, st>>>(l, atoms, perm, tiles, n_elem, key, count);
  return cudaGetLastError();
}

cudaError_t launch_cells_build(const CellLattice &l, const AtomD *atoms, const int *perm, int n_padded, int n_elem,
                               const int *key, const int *count, const int *run_begin, int *cursor, int *order,
                               AtomD *out, int n_slots, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(out, 0, n_slots * sizeof(AtomD), st);  // padding: weight 0
  if (e != cudaSuccess || n_padded <= 0) return e;
  const unsigned grid = (unsigned)((n_padded + 255) / 256);
  cells_order_kernel<<<grid, 256, 0, st>>>(perm, n_padded, key, run_begin, cursor, order);
  cells_place_kernel<<<grid, 256, 0, st>>>(l, atoms, perm, n_padded, n_elem, key, count, run_begin, order, out);
  return cudaGetLastError();
}

}  // namespace spsim
