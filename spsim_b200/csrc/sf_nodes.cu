// Structure-factor kernel on the nodes of coarse grids (sm_100a).
#include "sf_kernels.cuh"

namespace spsim {

// Test hook of the bounded waits, as g_copy_stall in sf_kernels.cu.
__device__ int g_nodes_copy_stall = 0;

cudaError_t set_nodes_copy_stall(int on) {
  const int v = on ? 1 : 0;
  return cudaMemcpyToSymbol(g_nodes_copy_stall, &v, sizeof(int));
}

// ---------------------------------------------------------------------------
// The quad form on the nodes of a coarse grid (coarse_kernels.cuh).  Nodes are
// too far apart for FP32 steps, so all eight points of a thread (two runs of
// four neighbours, as its two quads) take their own FP64 phase, and the NODE
// polynomials, with the fewer points' time to spare, one more coefficient than
// DHALF.  There are few nodes, so the warps of a CTA share one tile of 256 and
// take its atoms in turn, groups of eight, adding their FP64 sums at the end
// of the item: against 1,024 nodes per CTA that makes a work item a quarter as
// long (the launch's tail) and lets a grid of some hundred nodes use the GPU.
// Bound by the FMA and FP64 pipes, which add up: 14.6 FP32 and 3 FP64 lane
// operations per term allow 1.75e12 terms/s.  Measured on 50,000 atoms x 26,244
// nodes: 1.29e12 (1.27e12 with the sign on the ALU pipe, 1.24e12 with a full /
// empty barrier pair per stage instead of the CTA barrier, 1.28e12 with three
// CTAs per SM; FP32 sums of 16 atoms take the same time and have half as much
// error again).  On cells (kCellSizes in capi.cu) the runs of an element are
// short: 1.0e12 on 65 cells of 770 atoms x 71^2 nodes and on 65 of 308 x 22^2,
// from the padding to groups, the flushes and the items' starts (not from their
// latency: the next item's number and the form factors read ahead change
// nothing).
constexpr int NODE_THREADS = 128;
constexpr int NODE_TILE = SF_NODES_TILE;  // nodes per work item: 8 per lane
static_assert(NODE_TILE == 256, "eight nodes per lane");
// Tiles in flight: those of most work items of a cell at once, so that its warps
// meet only at the item's end (as many as static shared memory holds).
constexpr int NODE_STAGES = 7;

template <bool PERB, bool FIXW>
__global__ void __launch_bounds__(NODE_THREADS, 1) sf_dquad_nodes_kernel(
    const SfPattern *__restrict__ pats, const WorkItem *__restrict__ items, int n_items, int *__restrict__ queue,
    int *__restrict__ err, uint32_t m31) {
  constexpr int P = 8, NP = P / 2, WARPS = NODE_THREADS / 32;
  __shared__ __align__(128) float4 ring[NODE_STAGES][2 * TILE_ATOMS];
  __shared__ __align__(16) double2 sacc[P * NODE_THREADS];  // per-thread FP64 sums of the current work item
  __shared__ __align__(8) uint64_t full_bar[NODE_STAGES];
  __shared__ int s_item;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < NODE_STAGES; ++s) mbar_init(&full_bar[s], 1);
    fence_barrier_init();
  }
  __syncthreads();

  uint32_t g_issue = 0, g_cons = 0;
  const bool stall = g_nodes_copy_stall != 0;
  const long long kWaitCycles = stall ? kStallWaitCycles : kWaitCyclesDefault;
  const double M52 = 6755399441055744.0;  // 1.5 * 2^52
  constexpr double kQScale = FIXW ? 2.0 : 1.0;
  constexpr bool LOGW = PERB && FIXW;  // the weight folded into the exponent, as in sf_dquad_kernel

  for (;;) {
    if (tid == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= n_items) break;
    const WorkItem wi = items[it];
    const SfPattern &pt = pats[wi.pattern];
    const long long npix = pt.npix;
    const AtomD *__restrict__ atomsd = pt.atomsd;
    const TileDesc *__restrict__ tiles = pt.tiles;
    const int cell = pt.cell_tiles ? wi.pixel_tile / pt.cell_tiles : 0;
    double2 *__restrict__ acc = pt.acc + cell * npix;

    // node i of this lane: pix0 + 128 (i / 4) + i % 4
    const long long pix0 = (long long)(wi.pixel_tile - cell * pt.cell_tiles) * NODE_TILE + 4 * lane;
    double qx[P], qy[P], qz[P];
    float s2n[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const long long p = pix0 + 128 * (i / 4) + i % 4;
      double q[3] = {0.0, 0.0, 0.0};
      if (p < npix) load_q(pt, p, q);
      qx[i] = kQScale * q[0];
      qy[i] = kQScale * q[1];
      qz[i] = kQScale * q[2];
      s2n[i] = (float)(-0.25 * (q[0] * q[0] + q[1] * q[1] + q[2] * q[2]) * 1e-20 * pt.s2scale * 1.4426950408889634);
    }
    float2 shc[NP], slc[NP], shs[NP], sls[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) shc[j] = slc[j] = shs[j] = sls[j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < P; ++i) sacc[i * NODE_THREADS + tid] = make_double2(0.0, 0.0);

    const int k0 = wi.k0, k1 = wi.k1;
    if (tid == 0) {
      for (int k = k0; k < k1 && k < k0 + NODE_STAGES; ++k) {
        const TileDesc td = tiles[k];
        const uint32_t st = g_issue % NODE_STAGES;
        const uint32_t bytes = (uint32_t)td.count * (uint32_t)sizeof(AtomD);
        mbar_arrive_expect_tx(&full_bar[st], bytes);
        if (!(stall && g_issue == 0))  // the stall hook skips the CTA's first copy
          bulk_copy_g2s(&ring[st][0], atomsd + td.atom_begin, bytes, &full_bar[st]);
        ++g_issue;
      }
    }

    bool failed = false;
    int groups = 0;  // of the tiles before, so that the warps' shares of a run's last groups even out
    for (int k = k0; k < k1; ++k) {
      const uint32_t st = g_cons % NODE_STAGES;
      const uint32_t par = (g_cons / NODE_STAGES) & 1u;
      // a copy that did not come: this item's rest is passed over, and the CTA returns at its end
      if (!failed) failed = !mbar_wait_bounded(&full_bar[st], par, kWaitCycles);
      const TileDesc td = tiles[k];
      const float4 *__restrict__ ta = ring[st];
      // this warp's groups of eight atoms, in FP32 sums of four: of bright nodes'
      // sums, all of one sign, the rounding errors grow with the sum
      const int end = failed ? 0 : td.count;
      for (int a = ATOM_GROUP * ((warp - groups) & (WARPS - 1)); a < end; a += ATOM_GROUP * WARPS)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float2 bc[NP], bs[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) bc[j] = bs[j] = make_float2(0.f, 0.f);
#pragma unroll
        for (int g = 0; g < ATOM_GROUP / 2; ++g) {
          const int at = a + ATOM_GROUP / 2 * half + g;
          const float4 d0 = ta[2 * at], d1 = ta[2 * at + 1];
          const double rx = __hiloint2double(__float_as_int(d0.y), __float_as_int(d0.x));
          const double ry = __hiloint2double(__float_as_int(d0.w), __float_as_int(d0.z));
          const double rz = __hiloint2double(__float_as_int(d1.y), __float_as_int(d1.x));
          const float W = d1.z;
          const float lw = LOGW ? lg2_approx(fabsf(W)) : 0.0f;
          const double wbase = LOGW && W < 0.0f ? PHASE_WORD_BASE_HALF + 1.0 : PHASE_WORD_BASE_HALF;
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            float y[2], w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int i = 2 * j + h;
              uint32_t kb;
              if (FIXW) {
                const double t = phase_word(qx[i], qy[i], qz[i], rx, ry, rz, wbase);
                reduce_phase_word<PREC_MODE_POLY>(t, y[h], kb);
              } else {
                double u = qx[i] * rx;
                u = fma(qy[i], ry, u);
                u = fma(qz[i], rz, u);
                const double t = fma(u, 2.0, M52);
                y[h] = __double2float_rn(fma(t - M52, -0.5, u));
                kb = (uint32_t)__double2loint(t);
              }
              w[h] = LOGW ? ex2_approx(fmaf(d1.w, s2n[i], lw)) : PERB ? W * ex2_approx(d1.w * s2n[i]) : W;
              w[h] = sign_by_parity(w[h], kb, m31);
            }
            const float2 yy = FIXW ? mul2(make_float2(y[0], y[1]), f2(word_to_phase<PREC_MODE_POLY>()))
                                   : make_float2(y[0], y[1]);
            float2 S, C;
            sincos_node_poly2(yy, S, C);
            const float2 ws = make_float2(w[0], w[1]);
            bc[j] = fma2(ws, C, bc[j]);
            bs[j] = fma2(ws, S, bs[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          ff_accumulate2(shc[j], slc[j], bc[j]);
          ff_accumulate2(shs[j], sls[j], bs[j]);
        }
      }
      if (td.last || k == k1 - 1) {
        const double *__restrict__ ffe = pt.ff + (long long)td.elem * npix;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = 2 * j + h;
            const long long p = pix0 + 128 * (i / 4) + i % 4;
            if (p < npix) {
              const double f = ffe[p];
              const double re = h ? (double)shc[j].y + (double)slc[j].y : (double)shc[j].x + (double)slc[j].x;
              const double sm = h ? (double)shs[j].y + (double)sls[j].y : (double)shs[j].x + (double)sls[j].x;
              double2 v = sacc[i * NODE_THREADS + tid];
              v.x = fma(f, re, v.x);
              v.y = fma(-f, sm, v.y);
              sacc[i * NODE_THREADS + tid] = v;
            }
          }
          shc[j] = slc[j] = shs[j] = sls[j] = make_float2(0.f, 0.f);
        }
      }
      groups += td.count / ATOM_GROUP;
      ++g_cons;
      if (k + NODE_STAGES >= k1) continue;
      __syncthreads();
      if (tid == 0 && !failed) {
        const TileDesc tn = tiles[k + NODE_STAGES];
        const uint32_t bytes = (uint32_t)tn.count * (uint32_t)sizeof(AtomD);
        mbar_arrive_expect_tx(&full_bar[st], bytes);
        bulk_copy_g2s(&ring[st][0], atomsd + tn.atom_begin, bytes, &full_bar[st]);
        ++g_issue;
      }
    }
    if (__syncthreads_or(failed)) {
      if (tid == 0) {
        atomicOr(err, 1);
        for (uint32_t g = g_issue > NODE_STAGES ? g_issue - NODE_STAGES : 0; g < g_issue; ++g)
          mbar_wait_bounded(&full_bar[g % NODE_STAGES], (g / NODE_STAGES) & 1u, kWaitCycles);
      }
      return;
    }
    // item done: the warps' sums of each node added, one write per node (a plain
    // store when the item covers every atom tile of the molecule)
    const bool whole = k0 == 0 && k1 == pt.n_tiles;
#pragma unroll
    for (int r = 0; r < P / WARPS; ++r) {
      const int i = warp * (P / WARPS) + r;
      const long long p = pix0 + 128 * (i / 4) + i % 4;
      double2 v = sacc[i * NODE_THREADS + lane];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) {
        const double2 u = sacc[i * NODE_THREADS + 32 * w + lane];
        v.x += u.x;
        v.y += u.y;
      }
      if (p < npix) {
        if (whole) {
          acc[p] = v;
        } else {
          atomicAdd(&acc[p].x, v.x);
          atomicAdd(&acc[p].y, v.y);
        }
      }
    }
    __syncthreads();
  }
}

// FP64 term of the nodes: cos and sin / y of 2 pi y, |y| <= 1/4, z = y^2, and the
// weight's exponential.  FULL (coarse_digits in capi.cu): to the rounding (FULL64 and
// exp2_full, seven more operations); else to 1.7e-11 for FP32 results.
template <bool FULL>
__device__ __forceinline__ void node64_sincos(double z, double &ps, double &pc) {
  if (FULL) {
    ps = fma(z, SPSIM_FULL64_S8, SPSIM_FULL64_S7);
    pc = fma(z, SPSIM_FULL64_C8, SPSIM_FULL64_C7);
    ps = fma(z, ps, SPSIM_FULL64_S6);
    pc = fma(z, pc, SPSIM_FULL64_C6);
    ps = fma(z, ps, SPSIM_FULL64_S5);
    pc = fma(z, pc, SPSIM_FULL64_C5);
    ps = fma(z, ps, SPSIM_FULL64_S4);
    pc = fma(z, pc, SPSIM_FULL64_C4);
    ps = fma(z, ps, SPSIM_FULL64_S3);
    pc = fma(z, pc, SPSIM_FULL64_C3);
    ps = fma(z, ps, SPSIM_FULL64_S2);
    pc = fma(z, pc, SPSIM_FULL64_C2);
    ps = fma(z, ps, SPSIM_FULL64_S1);
    pc = fma(z, pc, SPSIM_FULL64_C1);
    ps = fma(z, ps, SPSIM_FULL64_S0);
    pc = fma(z, pc, SPSIM_FULL64_C0);
  } else {
    ps = fma(z, SPSIM_NODE64_S5, SPSIM_NODE64_S4);
    pc = fma(z, SPSIM_NODE64_C6, SPSIM_NODE64_C5);
    ps = fma(z, ps, SPSIM_NODE64_S3);
    pc = fma(z, pc, SPSIM_NODE64_C4);
    ps = fma(z, ps, SPSIM_NODE64_S2);
    pc = fma(z, pc, SPSIM_NODE64_C3);
    ps = fma(z, ps, SPSIM_NODE64_S1);
    pc = fma(z, pc, SPSIM_NODE64_C2);
    ps = fma(z, ps, SPSIM_NODE64_S0);
    pc = fma(z, pc, SPSIM_NODE64_C1);
    pc = fma(z, pc, SPSIM_NODE64_C0);
  }
}

// The same sum in FP64 throughout, phases by rounding.  B200's FP64 pipe runs at
// half the FP32 rate, and without the split phase and the compensated sums a
// term is 21 operations, so this takes 1.8 times as long as the FP32 kernel
// (7.2e11 terms/s on 50,000 atoms x 26,244 nodes, P = 4; 80 % of the pipe).  It
// runs
//   - in FP64 (FULL: 28 operations, 5.6e11 terms/s on 50,000 atoms in cells of
//     1024^2 pixels where the shorter polynomials take 6.5e11), where amplitudes
//     fall far (coarse_digits in capi.cu), and for molecules rewritten on the
//     device, that is in refinements: a node's rounding error goes into all the pixels around it
//     alike, and the gradient of a loss adds it up where the pixels' own errors
//     would average out (up to 6 times the gradient's error on a heavily
//     oversampled detector);
//   - for small grids, which latency bounds: with P = 2 a work item is 64 nodes
//     (1,000 atoms x 340 nodes: 12 us against 17 us in FP32; 5,000 x 840 even).
template <int P, bool PERB, bool FULL>
__global__ void __launch_bounds__(NODE_THREADS, 1) sf_nodes64_kernel(const SfPattern *__restrict__ pats,
                                                                  const WorkItem *__restrict__ items, int n_items,
                                                                  int *__restrict__ queue, int *__restrict__ err) {
  constexpr int WARPS = NODE_THREADS / 32;
  __shared__ __align__(128) float4 ring[RING_STAGES][2 * TILE_ATOMS];
  __shared__ __align__(16) double2 sacc[P * NODE_THREADS];
  __shared__ __align__(8) uint64_t full_bar[RING_STAGES];
  __shared__ int s_item;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < RING_STAGES; ++s) mbar_init(&full_bar[s], 1);
    fence_barrier_init();
  }
  __syncthreads();

  uint32_t g_issue = 0, g_cons = 0;
  const bool stall = g_nodes_copy_stall != 0;
  const long long kWaitCycles = stall ? kStallWaitCycles : kWaitCyclesDefault;
  const double M52 = 6755399441055744.0;  // 1.5 * 2^52

  for (;;) {
    if (tid == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= n_items) break;
    const WorkItem wi = items[it];
    const SfPattern &pt = pats[wi.pattern];
    const long long npix = pt.npix;
    const AtomD *__restrict__ atomsd = pt.atomsd;
    const TileDesc *__restrict__ tiles = pt.tiles;
    const int cell = pt.cell_tiles ? wi.pixel_tile / pt.cell_tiles : 0;
    double2 *__restrict__ acc = pt.acc + cell * npix;

    // node i of this lane: pix0 + 32 i
    const long long pix0 = (long long)(wi.pixel_tile - cell * pt.cell_tiles) * (32 * P) + lane;
    double qx[P], qy[P], qz[P];
    double s2n[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      double q[3] = {0.0, 0.0, 0.0};
      if (pix0 + 32 * i < npix) load_q(pt, pix0 + 32 * i, q);
      qx[i] = q[0];
      qy[i] = q[1];
      qz[i] = q[2];
      s2n[i] = -0.25 * (q[0] * q[0] + q[1] * q[1] + q[2] * q[2]) * 1e-20 * pt.s2scale * 1.4426950408889634;
    }
    double fre[P], fim[P], ec[P], es[P];  // the item's sums, and the current element's
#pragma unroll
    for (int i = 0; i < P; ++i) fre[i] = fim[i] = ec[i] = es[i] = 0.0;

    const int k0 = wi.k0, k1 = wi.k1;
    if (tid == 0) {
      for (int k = k0; k < k1 && k < k0 + RING_STAGES; ++k) {
        const TileDesc td = tiles[k];
        const uint32_t st = g_issue % RING_STAGES;
        const uint32_t bytes = (uint32_t)td.count * (uint32_t)sizeof(AtomD);
        mbar_arrive_expect_tx(&full_bar[st], bytes);
        if (!(stall && g_issue == 0))  // the stall hook skips the CTA's first copy
          bulk_copy_g2s(&ring[st][0], atomsd + td.atom_begin, bytes, &full_bar[st]);
        ++g_issue;
      }
    }

    for (int k = k0; k < k1; ++k) {
      const uint32_t st = g_cons % RING_STAGES;
      const uint32_t par = (g_cons / RING_STAGES) & 1u;
      const bool ok = mbar_wait_bounded(&full_bar[st], par, kWaitCycles);
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {
          atomicOr(err, 1);
          for (uint32_t g = g_cons; g < g_issue; ++g)
            mbar_wait_bounded(&full_bar[g % RING_STAGES], (g / RING_STAGES) & 1u, kWaitCycles);
        }
        return;
      }
      const TileDesc td = tiles[k];
      const float4 *__restrict__ ta = ring[st];
#pragma unroll 2
      for (int a = warp; a < td.count; a += WARPS) {
        const float4 d0 = ta[2 * a], d1 = ta[2 * a + 1];
        const double rx = __hiloint2double(__float_as_int(d0.y), __float_as_int(d0.x));
        const double ry = __hiloint2double(__float_as_int(d0.w), __float_as_int(d0.z));
        const double rz = __hiloint2double(__float_as_int(d1.y), __float_as_int(d1.x));
        const double W = d1.z, Bj = d1.w;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          double u = qx[i] * rx;
          u = fma(qy[i], ry, u);
          u = fma(qz[i], rz, u);
          const double t = fma(u, 2.0, M52);  // rint(2u) in the low bits
          const double y = fma(t - M52, -0.5, u);
          double w = PERB ? W * (FULL ? exp2_full(Bj * s2n[i]) : exp2_poly(Bj * s2n[i])) : W;
          w = __hiloint2double(__double2hiint(w) ^ (__double2loint(t) << 31), __double2loint(w));
          const double z = y * y;
          double ps, pc;
          node64_sincos<FULL>(z, ps, pc);
          ec[i] = fma(w, pc, ec[i]);
          es[i] = fma(w * y, ps, es[i]);
        }
      }
      if (td.last || k == k1 - 1) {
        const double *__restrict__ ffe = pt.ff + (long long)td.elem * npix;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          const double f = pix0 + 32 * i < npix ? ffe[pix0 + 32 * i] : 0.0;
          fre[i] = fma(f, ec[i], fre[i]);
          fim[i] = fma(-f, es[i], fim[i]);
          ec[i] = es[i] = 0.0;
        }
      }
      __syncthreads();
      if (tid == 0 && k + RING_STAGES < k1) {
        const TileDesc tn = tiles[k + RING_STAGES];
        const uint32_t bytes = (uint32_t)tn.count * (uint32_t)sizeof(AtomD);
        mbar_arrive_expect_tx(&full_bar[st], bytes);
        bulk_copy_g2s(&ring[st][0], atomsd + tn.atom_begin, bytes, &full_bar[st]);
        ++g_issue;
      }
      ++g_cons;
    }
#pragma unroll
    for (int i = 0; i < P; ++i) sacc[i * NODE_THREADS + tid] = make_double2(fre[i], fim[i]);
    __syncthreads();
    const bool whole = k0 == 0 && k1 == pt.n_tiles;
    for (int i = warp; i < P; i += WARPS) {
      double2 v = sacc[i * NODE_THREADS + lane];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) {
        const double2 u = sacc[i * NODE_THREADS + 32 * w + lane];
        v.x += u.x;
        v.y += u.y;
      }
      const long long p = pix0 + 32 * i;
      if (p < npix) {
        if (whole) {
          acc[p] = v;
        } else {
          atomicAdd(&acc[p].x, v.x);
          atomicAdd(&acc[p].y, v.y);
        }
      }
    }
    __syncthreads();
  }
}

// f(the kernel of node form `tile`), called with its arguments or queried for its occupancy
template <int P, typename F>
static void with_nodes64_p(bool perb, bool full, F f) {
  if (full)
    perb ? f(sf_nodes64_kernel<P, true, true>) : f(sf_nodes64_kernel<P, false, true>);
  else
    perb ? f(sf_nodes64_kernel<P, true, false>) : f(sf_nodes64_kernel<P, false, false>);
}
template <typename F>
static void with_nodes64(int tile, bool perb, bool full, F f) {
  tile == SF_NODES64_TILE ? with_nodes64_p<4>(perb, full, f) : with_nodes64_p<2>(perb, full, f);
}

cudaError_t launch_sf_nodes(int tile, bool perb, bool fixw, bool full, const SfPattern *pats, const WorkItem *items,
                            int n_items, int *queue, int *err, int grid, cudaStream_t st) {
  if (tile != SF_NODES_TILE)
    with_nodes64(tile, perb, full,
                 [&](auto kernel) { kernel<<<grid, NODE_THREADS, 0, st>>>(pats, items, n_items, queue, err); });
  else if (perb)
    fixw ? sf_dquad_nodes_kernel<true, true><<<grid, NODE_THREADS, 0, st>>>(pats, items, n_items, queue, err, 0x80000000u)
         : sf_dquad_nodes_kernel<true, false><<<grid, NODE_THREADS, 0, st>>>(pats, items, n_items, queue, err,
                                                                            0x80000000u);
  else
    fixw ? sf_dquad_nodes_kernel<false, true><<<grid, NODE_THREADS, 0, st>>>(pats, items, n_items, queue, err,
                                                                            0x80000000u)
         : sf_dquad_nodes_kernel<false, false><<<grid, NODE_THREADS, 0, st>>>(pats, items, n_items, queue, err,
                                                                             0x80000000u);
  return cudaGetLastError();
}

int sf_nodes_occupancy(int tile, bool perb, bool fixw, bool full) {
  int n = 0;
  if (tile != SF_NODES_TILE) {
    with_nodes64(tile, perb, full,
                 [&](auto kernel) { cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, NODE_THREADS, 0); });
    return n;
  }
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &n, perb ? (fixw ? sf_dquad_nodes_kernel<true, true> : sf_dquad_nodes_kernel<true, false>)
               : (fixw ? sf_dquad_nodes_kernel<false, true> : sf_dquad_nodes_kernel<false, false>),
      NODE_THREADS, 0);
  return n;
}

}  // namespace spsim
