// Cell moments of h(d) = Re sum_j w_j C_j e^{i gamma_j d}: host interface (k2_cells.cu).
//
// The offset scans and the per-peak polishes evaluate h at many offsets d of one point y, with
// C_j = 2 c_j e^{i gamma_j y}.  Split the zeros into cells of half width H in G = gamma / 2pi around
// centres G_c and put x_j = (G_j - G_c) / H in [-1, 1]:
//   h(d) = Re sum_c e^{2 pi i G_c d} sum_n M_cn (i kappa d)^n / n!,   kappa = 2 pi H,
//   M_cn = sum_{j in c} w_j C_j x_j^n.
// Every zero enters the moments once, whatever the number of offsets; with |kappa d| <= X the
// series cut after D1 terms is within X^D1 / D1! per unit of amplitude: 1 to 9 units of 2^-53 at the worst for the
// (X, D1) below, and less than one on average over a cell (the mean of |x|^D1 is 1 / (D1 + 1)).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "k2_internal.h"

namespace mb {

// |kappa d| bound for D1 series terms: X^D1 / D1! (the first dropped term, per unit amplitude)
//   D1 = 8,  X = 0.05: 9.7e-16    D1 = 16, X = 0.68: 1.0e-16    D1 = 11, X = 0.2: 5.1e-16
// at the cell's edge and the farthest offset.
constexpr double cell_x(int d1) { return d1 == 8 ? 0.05 : (d1 == 11 ? 0.2 : 0.68); }

int cell_peaks(int64_t P, int d1);      // points of one CTA of launch_moments_gauss
constexpr int CELL_MAX_W = 5;           // weight vectors of one moment pass
constexpr int CELL_D1 = 11;             // series terms of the polish paths

// Zero cells on the device: cell c holds the zeros [j0[c], j1[c]), centre ctr[c] 2^-16 in G.
struct Cells {
    int n = 0;                // cells in all
    int n_first = 0;          // cells of the first group (a prefix of the zeros; n if one group)
    int64_t half = 1;         // half width in units of 2^-16
    const int *j0 = nullptr, *j1 = nullptr;
    const int64_t *ctr = nullptr;
    double H() const { return (double)half * 0x1p-16; }
};

// A cell split planned on the host: up to two groups of zeros [a, b), one cell width.
struct CellPlan {
    int groups = 0;
    int64_t a[2], b[2], e0[2];
    int nc[2];
    int64_t half = 1;
    int cells() const { return groups == 2 ? nc[0] + nc[1] : nc[0]; }
};

// Plans the cells of the zeros [0, n) for offsets |d| <= R and D1 terms, at least min_cells where
// the zeros allow it; with 0 < split < n the zeros [0, split) form the first group.  false: the
// offsets reach so far that cells would be narrower than 2^-15 in G.
bool plan_cells(const Table &t, int64_t n, int64_t split, double R, int d1, int64_t min_cells, CellPlan &out);

// Device bytes of the plan's arrays, and the arrays themselves (buf: at least that, 256-aligned).
size_t cells_bytes(const CellPlan &p);
int build_cells(const Table &t, const CellPlan &p, void *buf, Cells &out, cudaStream_t s);

struct CellWeights {
    const double *w[CELL_MAX_W];
};

// Moments of P points (device arrays, delta may be null) over the cells.
// Gaussian weight exp(-k gamma^2): out[(p n + c) 2 D1 + q D1 + m], q = 0 real, 1 imaginary.
int launch_moments_gauss(const Table &t, const Cells &c, const uint64_t *vi, const uint64_t *vf, int64_t P, double k,
                         int d1, double *out, cudaStream_t s);
// nw <= CELL_MAX_W weight vectors, CELL_D1 terms: out[(((w P) + p) n + c) 2 CELL_D1 + q CELL_D1 + m];
// peak p is point sel[p] (p where sel is null).  One peak's moments have the same bits whatever P and
// nw are.
int launch_moments_weights(const Table &t, const Cells &c, const uint64_t *vi, const uint64_t *vf,
                           const double *delta, const int *sel, int64_t P, int nw, const CellWeights &w,
                           double *out, cudaStream_t s);

// The Taylor polish's grid stage on P peaks: power sums of w C u^m, u = gamma 1e-4, over taylor_chunks(n)
// chunks of the zeros [0, n) (edges n (c / n_chunk)^1.5: the first ones are the shortest, and may be empty), then h(ddy) = sum_m (-1)^m / (2m)! z^{2m} sum w Re C u^{2m}
// - sum_m (-1)^m / (2m+1)! z^{2m+1} sum w Im C u^{2m+1}, z = ddy 1e4, on the grid: h_unpol = h(0), h_pol and
// ddy_pol its first grid point of largest |h|.  work: taylor_work_bytes(P, n_chunk).
// The results of a peak have the same bits whatever P is.
int taylor_chunks(int64_t n);
size_t taylor_work_bytes(int64_t P, int n_chunk);
int launch_taylor_grid(const Table &t, const uint64_t *vi, const uint64_t *vf, const double *delta, int64_t P,
                       int64_t n, int n_chunk, const double *w, const double *grid, int n_grid, void *work,
                       double *h_unpol, double *h_pol, double *ddy_pol, cudaStream_t s);

// Offset pairs +-m step of one evaluation CTA, and the CTAs of a block of Bp points (pairs 0 .. Bp / 2).
constexpr int CSCAN_PAIRS = 128;
inline int64_t cell_scan_ctas(int64_t Bp) { return (Bp / 2 + CSCAN_PAIRS) / CSCAN_PAIRS; }

// out[p n_m + b Bp + i] = h at the offset (i - Bp / 2) step of point p NB + b, i < Bp, b < NB
// (Bp NB >= n_m; the moments are those of the P NB points).
int launch_cell_scan(const Table &t, const Cells &c, int d1, const double *M, int64_t P, int NB, int Bp, int64_t n_m,
                     uint64_t step_int, uint64_t step_frac, double *out, cudaStream_t s);

// Polishes of P peaks under nw weights from their moments (CELL_D1 terms): the three loops of
// k2_polish.cuh (PolishMode), outputs at [w * out_stride + p].
//
// Newton amplifies the rounding of its sums where h'' is small (up to 1e9 over six steps under a weight
// vector without decay).  Each path carries an estimate of that error, and a peak whose offset could
// differ by more than POLISH_SENSITIVE of the step clamp from the loops over the zeros is polished
// again by those loops themselves (the same bits), spread over the GPU.
// So is a peak where two offsets farther apart than the loop's last step have |h| closer than the two ways' roundings
// (POLISH_TIE of the cells' amplitude): two starts that end near one maximum, the second not fully converged.
constexpr double POLISH_SENSITIVE = 1e-10;
constexpr double POLISH_TIE = 2e-15;
struct CellPolishArgs {
    int mode;                  // PolishMode
    int64_t P;
    int nw;
    int64_t out_stride;
    const double *grid;        // POLISH_SINGLE: the ddy values
    int n_grid;                // POLISH_SINGLE: their number; POLISH_EVAL_FAST: grid_steps
    double half;               // POLISH_EVAL_FAST: grid half width
    const int *sel;            // POLISH_TOPK: point and output index of each peak, else null
    double *h_unpol, *h_pol, *ddy_pol;
};
// Cells whose moments of one peak fit shared memory (221 KB): the polish then reads them from there.
constexpr int CPOL_CELLS = 1200;
// Device bytes of the second pass's list for P x nw peaks (its terms are in t.redo).
size_t cell_polish_bytes(int64_t P, int nw);
// vi, vf, delta: the points (as for launch_moments_weights); w: the weights; work: cell_polish_bytes.  Waits
// for the stream once, for the number of peaks to polish again.  NO_ROOM: not even one of these peaks' terms fit.
int launch_cell_polish(Table &t, const Cells &c, const double *M, const CellPolishArgs &a, const uint64_t *vi,
                       const uint64_t *vf, const double *delta, int64_t n, const CellWeights &w, void *work,
                       cudaStream_t s);

// Sets the moment and scan kernels' shared-memory limits (once per device and context).
int cell_kernel_attributes();

}  // namespace mb
