// The per-peak polish contracts of search/path1_kernel_opt.py on the GPU:
//   compute_exact_mpfr_AB   (:71-91)   -> mb_exact_AB: A_j, B_j = 2 c_j e^{i gamma_j y} from the exact
//                                         128-bit phase (the reference rounds a 256-bit mpfr product)
//   polish_single_peak      (:94-147)  -> mb_polish_single_peak (A/B rows) and
//                                         mb_polish_single_exact (exact phase)
//   fast_polish_batch_blas  (:150-221) -> mb_fast_polish_batch (A/B rows) and
//                                         mb_fast_polish_exact (exact phase)
// and, for the search drivers' polish_peaks_with_weights (search/path1_eval_fast.cpp:58-143, whose
// A/B form is in k2_compat.cu), mb_polish_peaks_exact and mb_polish_peaks_weights.
// The exact-phase forms read the table and the peaks' 64.64 fixed-point v (+ delta).  They polish on moments
// over cells of zeros (k2_cells.h), which visit each zero once per peak; where the offsets reach too far for
// cells, or memory is short, over the zeros with (A, B) computed on the fly, or, under several weight
// vectors, from matrices built chunk by chunk.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "k2_cells.h"
#include "k2_polish.cuh"

namespace mb {
namespace {

// one cluster of POLISH_CLUSTER CTAs per peak: the grid stays within 2^31 - 1 CTAs
constexpr int64_t MAX_POLISH_PEAKS = (int64_t)1 << 26;

__global__ void exact_ab_kernel(ABExact src, int64_t n, int64_t p0, double *A, double *B) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int64_t p = p0 + blockIdx.y;
    const ABExact::Peak pk = src.peak(p);
    double a, b;
    src.at(pk, j, a, b);
    const size_t o = (size_t)blockIdx.y * n + j;
    A[o] = a;
    B[o] = b;
}

// numpy.linspace(-hw, hw, 2 steps + 1) value for value: arange(num) * step + start, last = stop.
std::vector<double> linspace_grid(double hw, int steps) {
    std::vector<double> g;
    if (steps <= 0) return g;
    const int num = 2 * steps + 1;
    const double start = -hw, step = (hw - start) / (double)(num - 1);
    g.resize(num);
    for (int i = 0; i < num; ++i) {
        volatile double t = (double)i * step;   // two roundings, as numpy does
        g[i] = t + start;
    }
    g[num - 1] = hw;
    return g;
}

// Indices of the `top` largest |h|, largest first; equal |h| in index order.
std::vector<int> top_indices(const double *h, int64_t P, int top) {
    std::vector<int> idx(P);
    std::iota(idx.begin(), idx.end(), 0);
    const int k = (int)std::min<int64_t>(top, P);
    std::partial_sort(idx.begin(), idx.begin() + k, idx.end(), [h](int a, int b) {
        const double x = std::fabs(h[a]), y = std::fabs(h[b]);
        return x > y || (x == y && a < b);
    });
    idx.resize(k);
    return idx;
}

int check_grid(const double *grid, int64_t n_grid, const char *who) {
    MB_CHECK_ARG(grid != nullptr && n_grid >= 1 && n_grid <= (1 << 20), "%s: n_grid=%lld", who, (long long)n_grid);
    for (int64_t i = 0; i < n_grid; ++i)
        MB_CHECK_ARG(std::isfinite(grid[i]), "%s: grid[%lld] is not finite", who, (long long)i);
    return MB_OK;
}

int check_peaks(const mb::Table &t, int64_t P, const uint64_t *vi, const uint64_t *vf, const double *delta,
                int64_t n_zeros, const char *who) {
    MB_CHECK_ARG(vi && vf, "%s: null candidate array", who);
    MB_CHECK_ARG(P >= 0 && P <= ((int64_t)1 << 30), "%s: P=%lld", who, (long long)P);
    MB_CHECK_ARG(n_zeros >= 0 && n_zeros <= t.n, "%s: n_zeros=%lld of %lld", who, (long long)n_zeros,
                 (long long)t.n);
    if (delta)
        for (int64_t p = 0; p < P; ++p)
            MB_CHECK_ARG(std::isfinite(delta[p]) && std::fabs(delta[p]) <= 65536.0,
                         "%s: delta[%lld]=%g must be finite with |delta| <= 2^16", who, (long long)p, delta[p]);
    return MB_OK;
}

int check_weights(const mb::Table &t, int slot, const char *who) {
    MB_CHECK_ARG(slot >= 0 && slot < (int)t.d_weights.size(), "%s: weight slot %d not registered", who, slot);
    return MB_OK;
}

// Candidates, grid, outputs and selection staged in the table's io buffer.
struct ExactStage {
    uint64_t *vi, *vf;
    double *delta, *grid, *hu, *hp, *dp;
    int *sel;
};

int stage_exact(Table &t, int64_t P, const uint64_t *vi, const uint64_t *vf, const double *delta,
                const double *grid, int64_t n_grid, int top, ExactStage &s) {
    const size_t need = 6 * ((size_t)P * 8 + 256) + ((size_t)n_grid * 8 + 256) + ((size_t)top * 4 + 256) + 256;
    MB_TRY(t.io.ensure(need));
    t.polish_redone = -1;
    char *p = (char *)t.io.p;
    s.vi = carve<uint64_t>(p, P);
    s.vf = carve<uint64_t>(p, P);
    s.delta = carve<double>(p, P);
    s.hu = carve<double>(p, P);
    s.hp = carve<double>(p, P);
    s.dp = carve<double>(p, P);
    s.grid = carve<double>(p, n_grid);
    s.sel = carve<int>(p, top);
    if (P <= 4096) {             // one copy for the three arrays (each small pageable copy costs microseconds)
        const size_t step = (size_t)(s.vf - s.vi);
        std::vector<uint64_t> h(3 * step, 0);
        std::memcpy(h.data(), vi, P * 8);
        std::memcpy(h.data() + step, vf, P * 8);
        if (delta) std::memcpy(h.data() + 2 * step, delta, P * 8);
        MB_CUDA(cudaMemcpyAsync(s.vi, h.data(), 3 * step * 8, cudaMemcpyHostToDevice, t.stream));
    } else {
        MB_CUDA(cudaMemcpyAsync(s.vi, vi, P * 8, cudaMemcpyHostToDevice, t.stream));
        MB_CUDA(cudaMemcpyAsync(s.vf, vf, P * 8, cudaMemcpyHostToDevice, t.stream));
        if (delta)
            MB_CUDA(cudaMemcpyAsync(s.delta, delta, P * 8, cudaMemcpyHostToDevice, t.stream));
        else
            MB_CUDA(cudaMemsetAsync(s.delta, 0, P * 8, t.stream));
    }
    if (n_grid > 0 && grid) MB_CUDA(cudaMemcpyAsync(s.grid, grid, n_grid * 8, cudaMemcpyHostToDevice, t.stream));
    return MB_OK;
}

// The three output arrays of P values, one copy where they lie together.
int fetch_outputs(cudaStream_t st, int64_t P, const double *hu, const double *hp, const double *dp, double *out_hu,
                  double *out_hp, double *out_dp) {
    const int64_t step = hp - hu;
    if (P <= 65536 && step >= P && step <= P + 32 && dp - hp == step) {
        std::vector<double> h(2 * step + P);
        MB_CUDA(cudaMemcpyAsync(h.data(), hu, h.size() * 8, cudaMemcpyDeviceToHost, st));
        MB_CUDA(cudaStreamSynchronize(st));
        std::memcpy(out_hu, h.data(), P * 8);
        std::memcpy(out_hp, h.data() + step, P * 8);
        std::memcpy(out_dp, h.data() + 2 * step, P * 8);
        return MB_OK;
    }
    MB_CUDA(cudaMemcpyAsync(out_hu, hu, P * 8, cudaMemcpyDeviceToHost, st));
    MB_CUDA(cudaMemcpyAsync(out_hp, hp, P * 8, cudaMemcpyDeviceToHost, st));
    MB_CUDA(cudaMemcpyAsync(out_dp, dp, P * 8, cudaMemcpyDeviceToHost, st));
    MB_CUDA(cudaStreamSynchronize(st));
    return MB_OK;
}

// ------------------------------------------------------------------ polishes on cell moments

// Whether v + delta stays in [0, 2^64) at every peak: the moments are taken at that sum as a 64.64 number, which
// would wrap (the loops over the zeros keep delta apart).
bool sums_in_range(int64_t P, const uint64_t *vi, const uint64_t *vf, const double *delta) {
    typedef unsigned __int128 u128;
    if (!delta) return true;
    for (int64_t p = 0; p < P; ++p) {
        const u128 v = (u128)vi[p] << 64 | vf[p], d = (u128)std::round(std::fabs(delta[p]) * 0x1p64);
        if (delta[p] < 0.0 ? v < d : v + d < v) return false;
    }
    return true;
}

constexpr size_t POLISH_MOMENT_BYTES = (size_t)256 << 20;

// Plans the cells of a polish whose offsets stay within R of the peaks: true where the polish on moments is not
// slower than the loops over the zeros.  At least 592 cells (two items per CTA slot) where they hold 64 zeros: few
// peaks then still fill the GPU.  Twice as many, and 32 zeros, for POLISH_TOPK, whose offsets converge: shorter
// running sums in the moments, without which its ddy are three times as far off as the loops' (6.9e-20 against
// 2.4e-20 rms on 87,292 zeros, now 1.9e-20).  The split and the choice depend on the zeros, R and the loop alone, so a
// peak's results do not depend on the others in the call, nor on the number of weight vectors.
//   Up to CPOL_CELLS cells (their moments fit shared memory) four zeros a cell are enough.
//   Above that a polish costs ~cells per peak and start, and 1 / cells of the peaks fit a pass of
// POLISH_MOMENT_BYTES, whose moment pass costs ~n however few they are: together ~cells^2 / n of the loops' cost, for
// five vectors (POLISH_EVAL_FAST) more than for one.  Measured, in ms (256 peaks x 5 vectors unless given):
//   EVAL_FAST 600,000 zeros, 19,900 cells 23.1 against 29.2, 29,800 cells 43.7 against 29.4, 78,000 cells 242 against
//             29; 2,325,572 zeros, 34,000 cells 79 against 122, 66,000 cells 237 against 120; 20,000 zeros, one peak and
//             vector, 2,300 cells 0.29 against 0.28, 3,600 cells 0.44 against 0.28
//   SINGLE    one peak: 20,000 zeros, 1,400 cells 0.55 against 0.72, 3,600 cells 1.5 against 0.74; 600,000 zeros,
//             29,800 cells 11.2 against 16.5, 78,000 cells 28.0 against 15.8
//   TOPK      25 peaks: 100,000 zeros, 2,000 cells 0.21 against 0.29, 5,700 cells 0.31 against 0.29
bool plan_polish(const Table &t, int64_t n, int64_t split, double R, int mode, CellPlan &cp) {
    if (n < 1 || !std::isfinite(R)) return false;
    const int64_t few = mode == POLISH_TOPK ? std::min<int64_t>(n / 32, 1184) : std::min<int64_t>(n / 64, 592);
    if (!plan_cells(t, n, split, R, CELL_D1, few, cp)) return false;
    const int64_t c = cp.cells();
    // one peak's moments under a full set of vectors stay within the workspace
    if (c * (2 * CELL_D1 * 8 * CELL_MAX_W) > (int64_t)POLISH_MOMENT_BYTES) return false;
    if (c <= std::max<int64_t>(64, std::min<int64_t>(n / 4, CPOL_CELLS))) return true;
    const double zeros = mode == POLISH_EVAL_FAST ? 8 : (mode == POLISH_SINGLE ? 13 : 18);
    const double square = mode == POLISH_EVAL_FAST ? 700 : 2500;
    return (double)c * std::max(zeros, (double)c / square) <= (double)n;
}

// Polishes the P peaks of stage s (or its P selected ones, a.sel) over the zeros [0, n) under the weight
// slots, outputs a.h_unpol etc. on the device: per chunk of peaks and up to CELL_MAX_W vectors, one moment
// pass over the zeros and the polish on the moments.  NO_ROOM (outputs partly written): the device has no room
// for the moments or the second pass, and the caller takes the loops over the zeros.
int polish_on_cells(Table &t, const ExactStage &s, int64_t P, int64_t n, int n_weights, const int *slots,
                    const CellPlan &cp, CellPolishArgs a) {
    const size_t cb = cells_bytes(cp), one = (size_t)cp.cells() * 2 * CELL_D1 * 8;     // per (peak, weight)
    const int wmax = std::min(n_weights, CELL_MAX_W);
    const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(P, (int64_t)(POLISH_MOMENT_BYTES / (one * wmax))));
    bool room;
    MB_TRY(t.moments.ensure((cb + 256) + ((size_t)chunk * wmax * one + 256) + cell_polish_bytes(chunk, wmax), &room));
    if (!room) return NO_ROOM;
    char *q = (char *)t.moments.p;
    void *cbuf = carve<char>(q, cb);
    double *M = carve<double>(q, (size_t)chunk * wmax * (one / 8));
    void *work = q;
    Cells cells;
    MB_TRY(build_cells(t, cp, cbuf, cells, t.stream));
    const CellPolishArgs all = a;
    t.polish_redone = 0;
    for (int64_t p0 = 0; p0 < P; p0 += chunk)
        for (int w0 = 0; w0 < n_weights; w0 += CELL_MAX_W) {
            const int64_t np = std::min(chunk, P - p0);
            const int nw = std::min(n_weights - w0, CELL_MAX_W);
            CellWeights w{};
            for (int i = 0; i < nw; ++i) w.w[i] = t.d_weights[slots[w0 + i]];
            const int *sel = all.sel ? all.sel + p0 : nullptr;
            const int64_t po = sel ? 0 : p0, o = (int64_t)w0 * all.out_stride + po;
            MB_TRY(launch_moments_weights(t, cells, s.vi + po, s.vf + po, s.delta + po, sel, np, nw, w, M, t.stream));
            a.P = np;
            a.nw = nw;
            a.sel = sel;
            a.h_unpol = all.h_unpol + o;
            a.h_pol = all.h_pol + o;
            a.ddy_pol = all.ddy_pol + o;
            MB_TRY(launch_cell_polish(t, cells, M, a, s.vi + po, s.vf + po, s.delta + po, n, w, work, t.stream));
        }
    return MB_OK;
}

// The farthest offset the loops of k2_polish.cuh reach: the grid's, plus every Newton step at its clamp.
double eval_fast_reach(double half, int steps) { return (steps > 0 ? std::fabs(half) : 0.0) + 6 * 1e-4; }
double single_reach(double hw, int steps) { return (steps > 0 ? std::fabs(hw) : 0.0) + 8 * 2e-5; }

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" int mb_exact_AB(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                           const double *delta, int64_t n_zeros, double *out_A, double *out_B) {
    MB_CHECK_ARG(h && out_A && out_B, "mb_exact_AB: null argument");
    Table &t = table_of(h);
    MB_TRY(check_peaks(t, P, v_int, v_frac, delta, n_zeros, "mb_exact_AB"));
    if (P == 0 || n_zeros == 0) return MB_OK;
    MB_TRY(device_guard(t.device));
    const size_t N = (size_t)n_zeros;
    // peaks per pass: A/B slabs within 2 GiB, grid.y within 65535
    const int64_t chunk = (int64_t)std::max<size_t>(
        1, std::min<size_t>({(size_t)P, ((size_t)1 << 31) / (16 * N), (size_t)65535}));
    ExactStage s;
    MB_TRY(stage_exact(t, P, v_int, v_frac, delta, nullptr, 0, 0, s));
    MB_TRY(t.work.ensure(2 * ((size_t)chunk * N * 8 + 256)));
    char *wp = (char *)t.work.p;
    double *d_A = carve<double>(wp, chunk * N), *d_B = carve<double>(wp, chunk * N);
    const ABExact src{view(t), s.vi, s.vf, s.delta};
    for (int64_t p0 = 0; p0 < P; p0 += chunk) {
        const int64_t np = std::min(chunk, P - p0);
        dim3 grid((unsigned)((N + 255) / 256), (unsigned)np);
        exact_ab_kernel<<<grid, 256, 0, t.stream>>>(src, n_zeros, p0, d_A, d_B);
        MB_CUDA(cudaGetLastError());
        MB_CUDA(cudaMemcpyAsync(out_A + p0 * N, d_A, np * N * 8, cudaMemcpyDeviceToHost, t.stream));
        MB_CUDA(cudaMemcpyAsync(out_B + p0 * N, d_B, np * N * 8, cudaMemcpyDeviceToHost, t.stream));
    }
    MB_CUDA(cudaStreamSynchronize(t.stream));
    return MB_OK;
}

extern "C" int mb_polish_single_peak(int64_t n_peaks, int64_t n_zeros, int64_t ld, const double *A, const double *B,
                                     const double *gamma, const double *w, double grid_hw, int grid_steps,
                                     double *out_h_unpol, double *out_h_pol, double *out_ddy_pol) {
    const char *who = "mb_polish_single_peak";
    MB_CHECK_ARG(n_peaks >= 0 && n_zeros >= 0 && ld >= n_zeros && grid_steps >= 0 && grid_steps <= (1 << 19),
                 "%s: bad sizes", who);
    if (n_peaks == 0) return MB_OK;
    MB_CHECK_ARG(A && B && gamma && w && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null array", who);
    MB_CHECK_ARG(std::isfinite(grid_hw), "%s: grid_hw is not finite", who);
    const std::vector<double> grid = linspace_grid(grid_hw, grid_steps);
    std::lock_guard<std::mutex> lock(scratch_mutex());
    const size_t N = (size_t)std::max<int64_t>(n_zeros, 1), G = std::max<size_t>(grid.size(), 1);
    const int64_t chunk = (int64_t)std::max<size_t>(1, std::min<size_t>((size_t)n_peaks, ((size_t)1 << 31) / (16 * N)));
    const size_t bytes = 2 * (N * 8 + 256) + (G * 8 + 256) + 2 * ((size_t)chunk * N * 8 + 256) +
                         3 * ((size_t)chunk * 8 + 256);
    void *base = nullptr;
    MB_TRY(scratch_buffer(bytes, &base));
    char *p = (char *)base;
    double *d_g = carve<double>(p, N), *d_w = carve<double>(p, N), *d_grid = carve<double>(p, G);
    double *d_A = carve<double>(p, chunk * N), *d_B = carve<double>(p, chunk * N);
    double *d_hu = carve<double>(p, chunk), *d_hp = carve<double>(p, chunk), *d_dp = carve<double>(p, chunk);
    cudaStream_t s = cudaStreamPerThread;
    if (n_zeros > 0) {
        MB_CUDA(cudaMemcpyAsync(d_g, gamma, n_zeros * 8, cudaMemcpyHostToDevice, s));
        MB_CUDA(cudaMemcpyAsync(d_w, w, n_zeros * 8, cudaMemcpyHostToDevice, s));
    }
    if (!grid.empty()) MB_CUDA(cudaMemcpyAsync(d_grid, grid.data(), grid.size() * 8, cudaMemcpyHostToDevice, s));
    for (int64_t p0 = 0; p0 < n_peaks; p0 += chunk) {
        const int64_t np = std::min(chunk, n_peaks - p0);
        if (n_zeros > 0) {
            MB_CUDA(cudaMemcpy2DAsync(d_A, n_zeros * 8, A + p0 * ld, ld * 8, n_zeros * 8, np, cudaMemcpyHostToDevice, s));
            MB_CUDA(cudaMemcpy2DAsync(d_B, n_zeros * 8, B + p0 * ld, ld * 8, n_zeros * 8, np, cudaMemcpyHostToDevice, s));
        }
        PolishArgs a{n_zeros, d_g, d_w, d_grid, (int)grid.size(), 0.0, nullptr, d_hu, d_hp, d_dp};
        peak_polish_kernel<ABMatrix, POLISH_SINGLE><<<(unsigned)(np * POLISH_CLUSTER), POLISH_THREADS, 0, s>>>(ABMatrix{d_A, d_B, n_zeros}, a);
        MB_CUDA(cudaGetLastError());
        MB_CUDA(cudaMemcpyAsync(out_h_unpol + p0, d_hu, np * 8, cudaMemcpyDeviceToHost, s));
        MB_CUDA(cudaMemcpyAsync(out_h_pol + p0, d_hp, np * 8, cudaMemcpyDeviceToHost, s));
        MB_CUDA(cudaMemcpyAsync(out_ddy_pol + p0, d_dp, np * 8, cudaMemcpyDeviceToHost, s));
    }
    MB_CUDA(cudaStreamSynchronize(s));
    return MB_OK;
}

extern "C" int mb_fast_polish_batch(int64_t n_peaks, int64_t n_zeros, const double *A, const double *B,
                                    const double *gamma, const double *w, const double *ddy_grid, int64_t n_grid,
                                    int top, double *out_h_unpol, double *out_h_pol, double *out_ddy_pol) {
    const char *who = "mb_fast_polish_batch";
    MB_CHECK_ARG(n_peaks >= 0 && n_zeros >= 0 && top >= 0 && top <= 65536, "%s: bad sizes", who);
    if (n_peaks == 0) return MB_OK;
    MB_CHECK_ARG(A && B && gamma && w && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null array", who);
    MB_TRY(check_grid(ddy_grid, n_grid, who));
    std::lock_guard<std::mutex> lock(scratch_mutex());
    const size_t N = (size_t)std::max<int64_t>(n_zeros, 1);
    const int64_t chunk = (int64_t)std::max<size_t>(1, std::min<size_t>((size_t)n_peaks, ((size_t)1 << 31) / (16 * N)));
    const int64_t nsel = std::min<int64_t>(top, n_peaks);
    const size_t bytes = 2 * (N * 8 + 256) + ((size_t)n_grid * 8 + 256) + 2 * ((size_t)chunk * N * 8 + 256) +
                         3 * ((size_t)n_peaks * 8 + 256);
    void *base = nullptr;
    MB_TRY(scratch_buffer(bytes, &base));
    char *p = (char *)base;
    double *d_g = carve<double>(p, N), *d_w = carve<double>(p, N), *d_grid = carve<double>(p, n_grid);
    double *d_A = carve<double>(p, chunk * N), *d_B = carve<double>(p, chunk * N);
    double *d_hu = carve<double>(p, n_peaks), *d_hp = carve<double>(p, n_peaks), *d_dp = carve<double>(p, n_peaks);
    cudaStream_t s = cudaStreamPerThread;
    if (n_zeros > 0) {
        MB_CUDA(cudaMemcpyAsync(d_g, gamma, n_zeros * 8, cudaMemcpyHostToDevice, s));
        MB_CUDA(cudaMemcpyAsync(d_w, w, n_zeros * 8, cudaMemcpyHostToDevice, s));
    }
    MB_CUDA(cudaMemcpyAsync(d_grid, ddy_grid, n_grid * 8, cudaMemcpyHostToDevice, s));
    for (int64_t p0 = 0; p0 < n_peaks; p0 += chunk) {
        const int64_t np = std::min(chunk, n_peaks - p0);
        if (n_zeros > 0) {
            MB_CUDA(cudaMemcpyAsync(d_A, A + p0 * N, np * N * 8, cudaMemcpyHostToDevice, s));
            MB_CUDA(cudaMemcpyAsync(d_B, B + p0 * N, np * N * 8, cudaMemcpyHostToDevice, s));
        }
        MomentArgs m{n_zeros, d_g, d_w, d_grid, (int)n_grid, d_hu + p0, d_hp + p0, d_dp + p0};
        taylor_moments_kernel<ABMatrix><<<(unsigned)(np * POLISH_CLUSTER), POLISH_THREADS, 0, s>>>(ABMatrix{d_A, d_B, n_zeros}, m);
        MB_CUDA(cudaGetLastError());
    }
    MB_TRY(fetch_outputs(s, n_peaks, d_hu, d_hp, d_dp, out_h_unpol, out_h_pol, out_ddy_pol));
    if (nsel == 0) return MB_OK;
    // exact Newton on the top peaks: their rows gathered into the first slab rows
    const std::vector<int> sel = top_indices(out_h_pol, n_peaks, (int)nsel);
    for (int64_t done = 0; done < nsel; done += chunk) {
        const int64_t np = std::min(chunk, nsel - done);
        for (int64_t r = 0; r < np; ++r) {
            const int64_t q = sel[done + r];
            if (n_zeros > 0) {
                MB_CUDA(cudaMemcpyAsync(d_A + r * N, A + q * N, N * 8, cudaMemcpyHostToDevice, s));
                MB_CUDA(cudaMemcpyAsync(d_B + r * N, B + q * N, N * 8, cudaMemcpyHostToDevice, s));
            }
            MB_CUDA(cudaMemcpyAsync(d_hu + r, out_h_unpol + q, 8, cudaMemcpyHostToDevice, s));
            MB_CUDA(cudaMemcpyAsync(d_dp + r, out_ddy_pol + q, 8, cudaMemcpyHostToDevice, s));
        }
        PolishArgs a{n_zeros, d_g, d_w, nullptr, 0, 0.0, nullptr, d_hu, d_hp, d_dp};
        peak_polish_kernel<ABMatrix, POLISH_TOPK><<<(unsigned)(np * POLISH_CLUSTER), POLISH_THREADS, 0, s>>>(ABMatrix{d_A, d_B, n_zeros}, a);
        MB_CUDA(cudaGetLastError());
        std::vector<double> hp(np), dp(np);
        MB_CUDA(cudaMemcpyAsync(hp.data(), d_hp, np * 8, cudaMemcpyDeviceToHost, s));
        MB_CUDA(cudaMemcpyAsync(dp.data(), d_dp, np * 8, cudaMemcpyDeviceToHost, s));
        MB_CUDA(cudaStreamSynchronize(s));
        for (int64_t r = 0; r < np; ++r) {
            out_h_pol[sel[done + r]] = hp[r];
            out_ddy_pol[sel[done + r]] = dp[r];
        }
    }
    return MB_OK;
}

extern "C" int mb_polish_single_exact(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                      const double *delta, int64_t n_zeros, int weight_slot, double grid_hw,
                                      int grid_steps, double *out_h_unpol, double *out_h_pol, double *out_ddy_pol) {
    const char *who = "mb_polish_single_exact";
    MB_CHECK_ARG(h && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null argument", who);
    MB_CHECK_ARG(P <= MAX_POLISH_PEAKS, "%s: P=%lld above %lld peaks per call", who, (long long)P,
                 (long long)MAX_POLISH_PEAKS);
    Table &t = table_of(h);
    MB_TRY(check_peaks(t, P, v_int, v_frac, delta, n_zeros, who));
    MB_TRY(check_weights(t, weight_slot, who));
    MB_CHECK_ARG(grid_steps >= 0 && grid_steps <= (1 << 19) && std::isfinite(grid_hw), "%s: bad grid", who);
    if (P == 0) return MB_OK;
    MB_TRY(device_guard(t.device));
    const std::vector<double> grid = linspace_grid(grid_hw, grid_steps);
    ExactStage s;
    MB_TRY(stage_exact(t, P, v_int, v_frac, delta, grid.data(), (int64_t)grid.size(), 0, s));
    CellPlan cp;
    if (sums_in_range(P, v_int, v_frac, delta) &&
        plan_polish(t, n_zeros, 0, single_reach(grid_hw, grid_steps), POLISH_SINGLE, cp)) {
        const int st = polish_on_cells(t, s, P, n_zeros, 1, &weight_slot, cp,
                                       CellPolishArgs{POLISH_SINGLE, P, 1, P, s.grid, (int)grid.size(), 0.0, nullptr, s.hu,
                                                      s.hp, s.dp});
        if (st == MB_OK) return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
        if (st != NO_ROOM) return st;
        t.polish_redone = -1;
    }
    PolishArgs a{n_zeros, t.d_gamma, t.d_weights[weight_slot], s.grid, (int)grid.size(), 0.0, nullptr, s.hu, s.hp, s.dp};
    peak_polish_kernel<ABExact, POLISH_SINGLE><<<(unsigned)(P * POLISH_CLUSTER), POLISH_THREADS, 0, t.stream>>>(
        ABExact{view(t), s.vi, s.vf, s.delta}, a);
    MB_CUDA(cudaGetLastError());
    return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
}

extern "C" int mb_polish_peaks_exact(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                     const double *delta, int64_t n_zeros, int weight_slot, double grid_half_width,
                                     int grid_steps, double *out_h_unpol, double *out_h_pol, double *out_ddy_pol) {
    const char *who = "mb_polish_peaks_exact";
    MB_CHECK_ARG(h && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null argument", who);
    MB_CHECK_ARG(P <= MAX_POLISH_PEAKS, "%s: P=%lld above %lld peaks per call", who, (long long)P,
                 (long long)MAX_POLISH_PEAKS);
    Table &t = table_of(h);
    MB_TRY(check_peaks(t, P, v_int, v_frac, delta, n_zeros, who));
    MB_TRY(check_weights(t, weight_slot, who));
    MB_CHECK_ARG(grid_steps >= 0 && grid_steps <= (1 << 19) && std::isfinite(grid_half_width), "%s: bad grid", who);
    if (P == 0) return MB_OK;
    MB_TRY(device_guard(t.device));
    ExactStage s;
    MB_TRY(stage_exact(t, P, v_int, v_frac, delta, nullptr, 0, 0, s));
    CellPlan cp;
    if (sums_in_range(P, v_int, v_frac, delta) &&
        plan_polish(t, n_zeros, 4096, eval_fast_reach(grid_half_width, grid_steps), POLISH_EVAL_FAST, cp)) {
        const int st = polish_on_cells(t, s, P, n_zeros, 1, &weight_slot, cp,
                                       CellPolishArgs{POLISH_EVAL_FAST, P, 1, P, nullptr, grid_steps, grid_half_width,
                                                      nullptr, s.hu, s.hp, s.dp});
        if (st == MB_OK) return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
        if (st != NO_ROOM) return st;
        t.polish_redone = -1;
    }
    PolishArgs a{n_zeros, t.d_gamma, t.d_weights[weight_slot], nullptr, grid_steps, grid_half_width, nullptr,
                 s.hu, s.hp, s.dp};
    peak_polish_kernel<ABExact, POLISH_EVAL_FAST><<<(unsigned)(P * POLISH_CLUSTER), POLISH_THREADS, 0, t.stream>>>(
        ABExact{view(t), s.vi, s.vf, s.delta}, a);
    MB_CUDA(cudaGetLastError());
    return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
}

// polish_peaks_with_weights under several weight vectors, where the cells do not serve: the exact (A, B)
// of a chunk of peaks is written once to HBM (the reference's P x N matrices,
// search/eval_tech1_600k.py:216-273, with the exact phase of mb_exact_AB) and every weight's polish reads
// it, instead of recomputing each term's 128-bit phase and sine/cosine in every pass.  Chunks keep the
// matrices within AB_BUDGET bytes.
constexpr size_t AB_BUDGET = (size_t)4 << 30;

extern "C" int mb_polish_peaks_weights(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                       const double *delta, int64_t n_zeros, int n_weights, const int *weight_slots,
                                       double grid_half_width, int grid_steps, double *out_h_unpol,
                                       double *out_h_pol, double *out_ddy_pol) {
    const char *who = "mb_polish_peaks_weights";
    MB_CHECK_ARG(h && weight_slots && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null argument", who);
    MB_CHECK_ARG(n_weights >= 1 && n_weights <= 64, "%s: n_weights=%d (1..64)", who, n_weights);
    MB_CHECK_ARG(P <= MAX_POLISH_PEAKS, "%s: P=%lld above %lld peaks per call", who, (long long)P,
                 (long long)MAX_POLISH_PEAKS);
    Table &t = table_of(h);
    MB_TRY(check_peaks(t, P, v_int, v_frac, delta, n_zeros, who));
    for (int w = 0; w < n_weights; ++w) MB_TRY(check_weights(t, weight_slots[w], who));
    MB_CHECK_ARG(grid_steps >= 0 && grid_steps <= (1 << 19) && std::isfinite(grid_half_width), "%s: bad grid", who);
    if (P == 0) return MB_OK;
    if (n_zeros == 0) {                                  // nothing to hold: the per-weight form
        for (int w = 0; w < n_weights; ++w)
            MB_TRY(mb_polish_peaks_exact(h, P, v_int, v_frac, delta, 0, weight_slots[w], grid_half_width,
                                         grid_steps, out_h_unpol + w * P, out_h_pol + w * P, out_ddy_pol + w * P));
        return MB_OK;
    }
    MB_TRY(device_guard(t.device));
    ExactStage s;
    CellPlan cp;
    if (sums_in_range(P, v_int, v_frac, delta) &&
        plan_polish(t, n_zeros, 4096, eval_fast_reach(grid_half_width, grid_steps), POLISH_EVAL_FAST, cp)) {
        const size_t ob = (size_t)n_weights * P;
        MB_TRY(stage_exact(t, P, v_int, v_frac, delta, nullptr, (int64_t)(3 * ob), 0, s));
        double *hu = s.grid, *hp = hu + ob, *dp = hp + ob;       // outputs in the stage's grid array
        const int st = polish_on_cells(t, s, P, n_zeros, n_weights, weight_slots, cp,
                                       CellPolishArgs{POLISH_EVAL_FAST, P, n_weights, P, nullptr, grid_steps,
                                                      grid_half_width, nullptr, hu, hp, dp});
        if (st == MB_OK) return fetch_outputs(t.stream, (int64_t)ob, hu, hp, dp, out_h_unpol, out_h_pol, out_ddy_pol);
        if (st != NO_ROOM) return st;
    }
    MB_TRY(stage_exact(t, P, v_int, v_frac, delta, nullptr, 0, 0, s));
    // the matrices take at most AB_BUDGET bytes and at most half of the device's free memory
    size_t free_b = 0, total_b = 0;
    MB_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = std::min(AB_BUDGET, free_b / 2);
    const int64_t chunk =
        std::max<int64_t>(1, std::min<int64_t>({P, (int64_t)65535, (int64_t)(budget / (16 * (size_t)n_zeros))}));
    const size_t out_b = (size_t)n_weights * P * 8;
    DevBuf buf;
    MB_TRY(buf.ensure(2 * ((size_t)chunk * n_zeros * 8 + 256) + 3 * (out_b + 256)));
    char *q = (char *)buf.p;
    double *A = carve<double>(q, chunk * n_zeros);
    double *B = carve<double>(q, chunk * n_zeros);
    double *hu = carve<double>(q, (int64_t)n_weights * P);
    double *hp = carve<double>(q, (int64_t)n_weights * P);
    double *dp = carve<double>(q, (int64_t)n_weights * P);
    const ABExact ex{view(t), s.vi, s.vf, s.delta};
    cudaError_t e = cudaSuccess;
    for (int64_t c0 = 0; c0 < P && e == cudaSuccess; c0 += chunk) {
        const int64_t cn = std::min(chunk, P - c0);
        exact_ab_kernel<<<dim3((unsigned)((n_zeros + 255) / 256), (unsigned)cn), 256, 0, t.stream>>>(ex, n_zeros, c0,
                                                                                                     A, B);
        e = cudaGetLastError();
        for (int w = 0; w < n_weights && e == cudaSuccess; ++w) {
            const int64_t o = (int64_t)w * P + c0;
            PolishArgs a{n_zeros, t.d_gamma, t.d_weights[weight_slots[w]], nullptr, grid_steps, grid_half_width,
                         nullptr, hu + o, hp + o, dp + o};
            peak_polish_kernel<ABMatrix, POLISH_EVAL_FAST>
                <<<(unsigned)(cn * POLISH_CLUSTER), POLISH_THREADS, 0, t.stream>>>(ABMatrix{A, B, n_zeros}, a);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_h_unpol, hu, out_b, cudaMemcpyDeviceToHost, t.stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_h_pol, hp, out_b, cudaMemcpyDeviceToHost, t.stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_ddy_pol, dp, out_b, cudaMemcpyDeviceToHost, t.stream);
    const cudaError_t es = cudaStreamSynchronize(t.stream);       // nothing in flight before the free
    if (e == cudaSuccess) e = es;
    buf.release();
    if (e != cudaSuccess) {
        set_error("%s: %s", who, cudaGetErrorString(e));
        return MB_ERR_CUDA;
    }
    return MB_OK;
}

extern "C" int mb_table_polish_redone(const mb_table *h, int64_t *n_out) {
    MB_CHECK_ARG(h && n_out, "mb_table_polish_redone: null argument");
    *n_out = table_of(const_cast<mb_table *>(h)).polish_redone;
    return MB_OK;
}

extern "C" int mb_fast_polish_exact(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                    const double *delta, int64_t n_zeros, int weight_slot, const double *ddy_grid,
                                    int64_t n_grid, int top, double *out_h_unpol, double *out_h_pol,
                                    double *out_ddy_pol) {
    const char *who = "mb_fast_polish_exact";
    MB_CHECK_ARG(h && out_h_unpol && out_h_pol && out_ddy_pol, "%s: null argument", who);
    MB_CHECK_ARG(P <= MAX_POLISH_PEAKS, "%s: P=%lld above %lld peaks per call", who, (long long)P,
                 (long long)MAX_POLISH_PEAKS);
    Table &t = table_of(h);
    MB_TRY(check_peaks(t, P, v_int, v_frac, delta, n_zeros, who));
    MB_TRY(check_weights(t, weight_slot, who));
    MB_TRY(check_grid(ddy_grid, n_grid, who));
    MB_CHECK_ARG(top >= 0 && top <= 65536, "%s: top=%d", who, top);
    if (P == 0) return MB_OK;
    MB_TRY(device_guard(t.device));
    const int nsel = (int)std::min<int64_t>(top, P);
    ExactStage s;
    MB_TRY(stage_exact(t, P, v_int, v_frac, delta, ddy_grid, n_grid, nsel, s));
    const ABExact src{view(t), s.vi, s.vf, s.delta};
    const double *d_w = t.d_weights[weight_slot];
    const int n_chunk = taylor_chunks(n_zeros);
    const bool fold = sums_in_range(P, v_int, v_frac, delta);
    auto grid_stage = [&]() -> int {
        if (!fold) {
            const MomentArgs m{n_zeros, t.d_gamma, d_w, s.grid, (int)n_grid, s.hu, s.hp, s.dp};
            taylor_moments_kernel<ABExact><<<(unsigned)(P * POLISH_CLUSTER), POLISH_THREADS, 0, t.stream>>>(src, m);
            MB_CUDA(cudaGetLastError());
            return MB_OK;
        }
        int64_t pc = std::max<int64_t>(
            1, std::min<int64_t>(P, (int64_t)(POLISH_MOMENT_BYTES / taylor_work_bytes(1, n_chunk))));
        for (bool room = false; !room;) {                // fewer peaks a pass where memory is short
            MB_TRY(t.moments.ensure(taylor_work_bytes(pc, n_chunk), pc > 1 ? &room : nullptr));
            if (pc == 1) break;
            if (!room) pc = (pc + 1) / 2;
        }
        for (int64_t p0 = 0; p0 < P; p0 += pc)
            MB_TRY(launch_taylor_grid(t, s.vi + p0, s.vf + p0, s.delta + p0, std::min(pc, P - p0), n_zeros, n_chunk,
                                      d_w, s.grid, (int)n_grid, t.moments.p, s.hu + p0, s.hp + p0, s.dp + p0, t.stream));
        return MB_OK;
    };
    MB_TRY(grid_stage());
    if (nsel == 0) return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
    MB_CUDA(cudaMemcpyAsync(out_h_pol, s.hp, P * 8, cudaMemcpyDeviceToHost, t.stream));
    MB_CUDA(cudaStreamSynchronize(t.stream));
    const std::vector<int> sel = top_indices(out_h_pol, P, nsel);
    MB_CUDA(cudaMemcpyAsync(s.sel, sel.data(), nsel * sizeof(int), cudaMemcpyHostToDevice, t.stream));
    double reach = 4 * 1e-5;
    for (int64_t i = 0; i < n_grid; ++i) reach = std::max(reach, std::fabs(ddy_grid[i]) + 4 * 1e-5);
    CellPlan cp;
    if (fold && plan_polish(t, n_zeros, 0, reach, POLISH_TOPK, cp)) {
        const int st = polish_on_cells(t, s, nsel, n_zeros, 1, &weight_slot, cp,
                                       CellPolishArgs{POLISH_TOPK, nsel, 1, P, nullptr, 0, 0.0, s.sel, s.hu, s.hp, s.dp});
        if (st == MB_OK) return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
        if (st != NO_ROOM) return st;
        t.polish_redone = -1;
        MB_TRY(grid_stage());                            // the starts again: the cells' polish writes over them
    }
    PolishArgs a{n_zeros, t.d_gamma, d_w, nullptr, 0, 0.0, s.sel, s.hu, s.hp, s.dp};
    peak_polish_kernel<ABExact, POLISH_TOPK><<<(unsigned)(nsel * POLISH_CLUSTER), POLISH_THREADS, 0, t.stream>>>(src, a);
    MB_CUDA(cudaGetLastError());
    return fetch_outputs(t.stream, P, s.hu, s.hp, s.dp, out_h_unpol, out_h_pol, out_ddy_pol);
}
