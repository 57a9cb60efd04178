// Coarse detector grids (internal C++ interface).
//
// A pattern's centred amplitude A(x, y) = sum_e f_e sum_j w_j e^{-2 pi i q(x, y).(r_j - c)}
// over the pixel coordinates of a detector is smooth: no atom's phase turns
// faster than |dq/dx| |r - c|max cycles per pixel.  Where that is well below
// half a cycle, the sum is evaluated on a tensor grid of nodes instead of on
// every pixel and every pixel interpolates it: A = M_y A_nodes M_x^T in FP64.
// Along each axis of a flat detector the coordinate is the scattering angle
// atan(x / D), in which q moves along the Ewald sphere at (almost) constant
// speed; a spherical detector's q is linear in the pixel index.  The nodes are
// Chebyshev extreme points stretched towards equal spacing by
// x = asin(alpha xi) / asin(alpha) (Kosloff and Tal-Ezer, J. Comput. Phys. 104
// (1993) 457), so that little more than two of them per cycle are needed, and
// the interpolation is the barycentric formula in xi (Salzer; Berrut and
// Trefethen, SIAM Rev. 46 (2004) 501).
#pragma once

#include "sf_device.cuh"

namespace spsim {

// Pixel geometry of a detector q set, in the units of ewald_kernel.
struct DetGeom {
  int nx, ny;
  int spherical;
  double width, height, distance, cx, cy, ewald, fpx, fpy, px_size, py_size;
  double lift = 0.0;  // added to the nodes' q along the beam (launch_list_combine)
};

// One axis of a detector in the interpolation's coordinate X in [-1, 1]:
// (atan(x / D) - mid) / half of the pixel's position x on a flat detector,
// the scaled pixel index on a spherical one.
struct CoarseAxis {
  int n_pix, angular;
  double size, centre, distance, mid, half;
  int n;  // nodes
  double alpha, asin_alpha;
  // the points to interpolate to: the pixels, or (to_n > 0) another grid's nodes
  int to_n;
  double to_alpha, to_asin;
  int derivative;  // matrices of the interpolant's derivative by X instead
};

constexpr int COARSE_MAX_NODES = 1024;  // per axis

CoarseAxis coarse_axis(int n_pix, double size, double centre, double distance, bool spherical);
// Nodes along one axis for phases of at most c radians over half of it, pixels
// up to t detector distances off the beam axis and form factors falling as
// exp(-a X^2): a fit, from above, to the smallest node counts that interpolate
// every such function to 1e-8 of its maximum or, by digits, to 1e-12 or 1e-15
// (tests/test_coarse_grid.py restates it and measures the errors): FP32 results,
// FP32 results from FP64 sums, and FP64 results, whose phases' own rounding is
// larger (1e-16 of up to some thousand radians).
constexpr int COARSE_DIGITS_F32 = 8, COARSE_DIGITS_F64 = 12, COARSE_DIGITS_FULL = 15;
int coarse_node_count(double c, double t, double a, int digits);
void coarse_set_nodes(CoarseAxis &a, int n, int digits);

// What the interpolation of one pattern reads and writes beside its
// SfPattern of pixels.
struct CoarsePattern {
  const double2 *nodes;  // [nyn][nxn] centred amplitudes
  const double *mx;      // [nx][ldx]: weight of node column i for pixel column x at mx[x * ldx + coarse_slot(i)]
  const double *my;      // [ny][ldy]
  int nx, ny, nxn, nyn, ldx, ldy;
  double B;              // global B factor, applied per pixel
  double2 *out;          // centred pixel amplitudes (FP64) instead of F and I, or nullptr
  int parent;            // SfPattern of the points interpolated to
  // one cell of a molecule (launch_cells_build): its amplitudes, times the phase
  // of its centre `shift`, are added to sum on the pattern's own nodes
  double2 *sum;
  double shift[3];
};

__host__ __device__ inline int coarse_ld(int n) { return (n + 7) / 8 * 8; }

// Node q vectors [y.n * x.n][3] and both interpolation matrices of one
// detector, columns at coarse_slot; tx, ty: also their transposes, [nodes][coarse_ld(pixels)].
cudaError_t launch_coarse_tables(const DetGeom &g, const CoarseAxis &x, const CoarseAxis &y, double *q64, double *mx,
                                 double *my, cudaStream_t st, double *tx = nullptr, double *ty = nullptr);
// The patterns of one interpolation: either described one by one (pats, coarse)
// or, pats == nullptr, alike: pattern i reads one.nodes + i * nyn * nxn, takes
// the rotation rots + 9 i (or none) and writes F + i * npix and I + i * npix.
struct CoarseBatch {
  const SfPattern *pats;
  const CoarsePattern *coarse;
  CoarsePattern one;
  const double *q64, *rots;
  double center[3];
  float2 *F;
  float *I;
};
// Interpolates npat patterns in groups of as many as the strip buffer holds
// (strip_size complex values, at least max_nyn * max_nx).
// cells: the patterns are cells, added to the sums of the patterns they belong to.
cudaError_t launch_coarse_interp(const CoarseBatch &b, int npat, int max_nx, int max_ny, int max_nxn, int max_nyn,
                                 double2 *strip, long long strip_size, cudaStream_t st, bool cells = false);

// Patterns on a float HKL list that is a detector's own, rotated and rounded:
// q = R q_detector + delta with delta of a few float roundings.  The amplitudes
// on the detector's exact q, its derivatives along X and Y by the derivative
// matrices, and those at `lift` along the beam (a second node sum) give
// A + delta . grad A; the second order is below 1e-8 for the patterns admitted
// (phases of at most 100 cycles), as are the derivatives' own errors.
struct ListCombine {
  DetGeom g;
  CoarseAxis x, y;
  double rot[9];              // q_list ~ rot q_detector
  const float *hkl;           // [npix][3]
  const double2 *a, *ax, *ay, *lifted;  // centred amplitudes of the pixels, A, dA/dX, dA/dY and A(q + lift)
  double lift, B;
  double center[3];
  float2 *F;  // [npix] or nullptr
  float *I;
};
cudaError_t launch_list_combine(const ListCombine &c, long long p0, long long p1, cudaStream_t st);

// A molecule's atoms by cells, the Voronoi cells of a body-centred cubic
// lattice of constant a about the molecule's centre (the lattice whose cells'
// circumscribed sphere, of radius sqrt(5) / 4 a, is the smallest for their
// volume): cell ((sub * dim + z) * dim + y) * dim + x has its centre at
// a (x - reach + sub / 2, ...), dim = 2 reach + 1.
struct CellLattice {
  double a;
  int reach, dim;
};
// The count of atoms per (cell, element), and each atom's such index in key.
cudaError_t launch_cells_count(const CellLattice &l, const AtomD *atoms, const int *perm, const TileDesc *tiles,
                               int n_tiles, int n_elem, int *key, int *count, cudaStream_t st);
// The records of the cells: run_begin[key] is where (cell, element)'s begin, in
// the atoms' own order, their positions about the cell's centre.  cursor: as
// large as count, zero; order: n_slots, scratch.
cudaError_t launch_cells_build(const CellLattice &l, const AtomD *atoms, const int *perm, int n_padded, int n_elem,
                               const int *key, const int *count, const int *run_begin, int *cursor, int *order,
                               AtomD *out, int n_slots, cudaStream_t st);

// The adjoint of the interpolation: per pattern, from the forward's F and
// G = dL/d|F|^2 on the pixels to the amplitudes H on the nodes.
struct CoarseAdjoint {
  const float2 *F;      // [npat][npix]
  const float *G;       // [npat][npix]
  const double *q64, *rot;
  double center[3], B;
  long long npix;
  int nx, ny, nxn, nyn;
  const double *tx, *ty;  // transposed interpolation matrices
};
// Groups of `group` patterns at a time through H (group * npix complex values)
// and strip (group * nxn * ny).
cudaError_t launch_coarse_adjoint(const CoarseAdjoint &a, int npat, double2 *H, int group, double2 *strip,
                                  double2 *nodes, cudaStream_t st);

}  // namespace spsim
