// Grid scan: K2 at y_m = v + m step for m = m0 .. m0 + n_m - 1 (search/polish.py:50-72 evaluates
// h(y0 + m step) the same way in FP64 from phi_j = gamma_j y0 mod 2pi and dphi_j = gamma_j step
// mod 2pi).  Here step is a 64.64 fixed-point number and the phase of every grid point is exact:
//   frac(y_m G) = frac(frac(v G) + m frac(step G))     (128-bit words, mod 1)
// Each thread takes MPT consecutive grid points: one 128 x 32-bit product per zero gives the
// exact phase of the first, whose sine/cosine (FP64, quarter-turn polynomials) times the
// amplitude is rotated to the other MPT - 1 points by powers of (cos, sin)(2 pi frac(step G)) of
// that zero (the reference's angle addition, polish.py:60-66, gpu_mertens_stream.cu:324-356,
// anchored afresh at an exact phase every MPT points; each point at most four rotations from its
// anchor).  FP64 accumulation, deterministic reduction over zero chunks.
#include <algorithm>
#include <cmath>
#include <vector>

#include "k2_cells.h"
#include "k2_common.cuh"
#include "k2_internal.h"

namespace mb {
namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_MPT = 16;                    // grid points per thread (one exact anchor)
static_assert(SCAN_MPT == 16, "add_rotations16 covers 16 points");
constexpr int SCAN_TILE = 256;                  // zeros per staged tile
struct __align__(16) ZScan {
    uint64_t p_lo, p_hi;       // frac(v G) + psi, 2^-128 units
    uint64_t d_lo, d_hi;       // frac(step G), 2^-128 units
    double a;                  // 2 |c| exp(-k gamma^2)
    double rc[4], rs[4];       // cos, sin of 2^b 2 pi frac(step G), b = 0..3
    double pad;
};

// (c, s) rotated by the angle whose cosine and sine are (cd, sd)
MB_DEV void rot(double c, double s, double cd, double sd, double &oc, double &os) {
    oc = fma(c, cd, -s * sd);
    os = fma(s, cd, c * sd);
}

// acc[i] += Re((c + i s) e^{i i phi}) for i = 0..15, given (rc[b], rs[b]) = (cos, sin)(2^b phi):
// a rotation tree of depth 4 (z8 from z0, z4 and z12, then the even points, then the odd ones,
// which need only their cosine), so every point is at most four rotations from the exact anchor
// and the chains are independent.
MB_DEV void add_rotations16(double c0, double s0, const double (&rc)[4], const double (&rs)[4], double (&acc)[16]) {
    double c[16], s[16];
    c[0] = c0;
    s[0] = s0;
    rot(c[0], s[0], rc[3], rs[3], c[8], s[8]);
#pragma unroll
    for (int i = 0; i < 16; i += 8) rot(c[i], s[i], rc[2], rs[2], c[i + 4], s[i + 4]);
#pragma unroll
    for (int i = 0; i < 16; i += 4) rot(c[i], s[i], rc[1], rs[1], c[i + 2], s[i + 2]);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        acc[i] += c[i];
        acc[i + 1] += fma(c[i], rc[0], -s[i] * rs[0]);
    }
}

// (cos, sin)(2^b phi), b = 0..3, from (cos, sin)(phi) by repeated squaring
MB_DEV void rotation_powers(double cd, double sd, double (&rc)[4], double (&rs)[4]) {
    rc[0] = cd;
    rs[0] = sd;
#pragma unroll
    for (int b = 1; b < 4; ++b) {
        rc[b] = fma(rc[b - 1], rc[b - 1], -rs[b - 1] * rs[b - 1]);
        rs[b] = 2.0 * rc[b - 1] * rs[b - 1];
    }
}

// partial[((p * n_chunk) + chunk) * n_m + m]
__global__ void __launch_bounds__(SCAN_THREADS)
k2_scan_kernel(TabView t, const uint64_t *vi, const uint64_t *vf, uint64_t si, uint64_t sf, int64_t m0, int n_m,
               int64_t n_use, int64_t chunk, double k, double *partial) {
    __shared__ ZScan tile[SCAN_TILE];
    const int p = blockIdx.z;
    const int n_chunk = gridDim.y;
    const int mb = (blockIdx.x * SCAN_THREADS + threadIdx.x) * SCAN_MPT;     // first local grid index
    const uint64_t a_int = vi[p], a_frac = vf[p];
    double acc[SCAN_MPT];
#pragma unroll
    for (int i = 0; i < SCAN_MPT; ++i) acc[i] = 0.0;
    const int64_t z0 = (int64_t)blockIdx.y * chunk, z1 = min(z0 + chunk, n_use);
    const int64_t mstart = m0 + mb;                       // signed grid index of this thread's first point
    const uint32_t mabs = (uint32_t)(mstart < 0 ? -mstart : mstart);
    for (int64_t tb = z0; tb < z1; tb += SCAN_TILE) {
        __syncthreads();
        const int64_t j = tb + threadIdx.x;
        if (threadIdx.x < SCAN_TILE && j < z1) {
            ZScan r;
            uint64_t hi, lo;
            phase128_exact((uint32_t)a_frac, (uint32_t)(a_frac >> 32), (uint32_t)a_int, (uint32_t)(a_int >> 32),
                           t.g0[j], t.g1[j], t.g2[j], t.g3[j], t.g4[j], hi, lo);
            r.p_lo = lo;
            r.p_hi = hi + t.psi[j];
            phase128_exact((uint32_t)sf, (uint32_t)(sf >> 32), (uint32_t)si, (uint32_t)(si >> 32), t.g0[j], t.g1[j],
                           t.g2[j], t.g3[j], t.g4[j], hi, lo);
            r.d_lo = lo;
            r.d_hi = hi;
            const double g = t.gamma[j];
            r.a = 2.0 * t.alpha[j] * exp(-k * g * g);
            double cd, sd;
            sincospi(2.0 * s64_turns_to_f64(hi), &sd, &cd);   // ~1 ulp: errors add up over the rotations
            rotation_powers(cd, sd, r.rc, r.rs);
            r.pad = 0.0;
            tile[threadIdx.x] = r;
        }
        __syncthreads();
        if (mb >= n_m) continue;
        const int nt = (int)min((int64_t)SCAN_TILE, z1 - tb);
        for (int jj = 0; jj < nt; ++jj) {
            const ZScan z = tile[jj];
            // x = p + mstart d  (mod 2^128)
            uint64_t mlo = (uint64_t)mabs * z.d_lo;
            uint64_t mhi = __umul64hi((uint64_t)mabs, z.d_lo) + (uint64_t)mabs * z.d_hi;
            if (mstart < 0) {                          // negate (two's complement, 128 bits)
                mlo = ~mlo + 1;
                mhi = ~mhi + (mlo == 0 ? 1 : 0);
            }
            const uint64_t xlo = z.p_lo + mlo;
            const uint64_t xhi = z.p_hi + mhi + (xlo < mlo ? 1 : 0);
            double sn, cs;
            sincos_turns_quad(s64_turns_to_f64(xhi), sn, cs);
            add_rotations16(cs * z.a, sn * z.a, z.rc, z.rs, acc);
        }
    }
    if (mb < n_m) {
        double *o = partial + ((int64_t)p * n_chunk + blockIdx.y) * n_m;
#pragma unroll
        for (int i = 0; i < SCAN_MPT; ++i)
            if (mb + i < n_m) o[mb + i] = acc[i];
    }
}

// Small grids over many base points (the hit polish of the enumerators): n_split CTAs per base
// point, each over a contiguous share of the zeros (so a few hits still fill the GPU), each thread
// HIT_ZPT zeros per round; the shares' sums go to partial[(p n_split + s) n_m + m] and
// hit_reduce_kernel adds them in split order.  Per zero: the exact phase at the grid's first point and
// the exact increment per step; every HIT_MB points an exact anchor (FP64 sine/cosine of the
// 128-bit phase, times the amplitude), rotated to the points in between by powers of the
// increment's (cos, sin).  A block of HIT_MB points is summed over the thread's zeros, then over
// the warp by a fixed shuffle tree, and lane 0 adds it to its warp's row of shared accumulators
// (fixed order -> deterministic).
constexpr int HIT_THREADS = 256;
constexpr int HIT_MAX_M = 1024;
constexpr int HIT_ZPT = 2;
constexpr int HIT_MB = 16;
static_assert(HIT_MB == 16, "add_rotations16 and the anchor step (increment << 4) assume 16");

__global__ void __launch_bounds__(HIT_THREADS)
k2_hit_scan_kernel(TabView t, const uint64_t *vi, const uint64_t *vf, uint64_t si, uint64_t sf, int64_t m0, int n_m,
                   int64_t n_use, double k, int n_split, double *partial) {
    extern __shared__ double acc[];            // [HIT_THREADS / 32][n_m]
    const int64_t p = blockIdx.x / n_split;
    const int split = blockIdx.x - (int)(p * n_split);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < (HIT_THREADS / 32) * n_m; i += HIT_THREADS) acc[i] = 0.0;
    __syncthreads();
    const uint64_t a_int = vi[p], a_frac = vf[p];
    const uint32_t mabs = (uint32_t)(m0 < 0 ? -m0 : m0);
    constexpr int PER_ROUND = HIT_THREADS * HIT_ZPT;
    const int64_t rounds = (n_use + PER_ROUND - 1) / PER_ROUND;
    const int64_t r_end = rounds * (split + 1) / n_split;
    for (int64_t r = rounds * split / n_split; r < r_end; ++r) {
        uint64_t xlo[HIT_ZPT], xhi[HIT_ZPT], dlo[HIT_ZPT], dhi[HIT_ZPT];
        double a[HIT_ZPT], rc[HIT_ZPT][4], rs[HIT_ZPT][4];
#pragma unroll
        for (int z = 0; z < HIT_ZPT; ++z) {
            const int64_t j = r * PER_ROUND + z * HIT_THREADS + threadIdx.x;
            xlo[z] = xhi[z] = dlo[z] = dhi[z] = 0;
            a[z] = 0.0;
            double cd = 1.0, sd = 0.0;
            if (j < n_use) {
                uint64_t hi, lo;
                phase128_exact((uint32_t)a_frac, (uint32_t)(a_frac >> 32), (uint32_t)a_int, (uint32_t)(a_int >> 32),
                               t.g0[j], t.g1[j], t.g2[j], t.g3[j], t.g4[j], hi, lo);
                const uint64_t plo = lo, phi = hi + t.psi[j];
                phase128_exact((uint32_t)sf, (uint32_t)(sf >> 32), (uint32_t)si, (uint32_t)(si >> 32), t.g0[j],
                               t.g1[j], t.g2[j], t.g3[j], t.g4[j], dhi[z], dlo[z]);
                uint64_t mlo = (uint64_t)mabs * dlo[z];
                uint64_t mhi = __umul64hi((uint64_t)mabs, dlo[z]) + (uint64_t)mabs * dhi[z];
                if (m0 < 0) {
                    mlo = ~mlo + 1;
                    mhi = ~mhi + (mlo == 0 ? 1 : 0);
                }
                xlo[z] = plo + mlo;
                xhi[z] = phi + mhi + (xlo[z] < mlo ? 1 : 0);
                const double g = t.gamma[j];
                a[z] = 2.0 * t.alpha[j] * exp(-k * g * g);
                sincospi(2.0 * s64_turns_to_f64(dhi[z]), &sd, &cd);   // ~1 ulp: errors add up over the rotations
                // the anchors advance by HIT_MB steps: d <<= log2(HIT_MB) (mod 2^128)
                dhi[z] = (dhi[z] << 4) | (dlo[z] >> 60);
                dlo[z] <<= 4;
            }
            rotation_powers(cd, sd, rc[z], rs[z]);
        }
        for (int mb = 0; mb < n_m; mb += HIT_MB) {
            double v[HIT_MB];
#pragma unroll
            for (int i = 0; i < HIT_MB; ++i) v[i] = 0.0;
#pragma unroll
            for (int z = 0; z < HIT_ZPT; ++z) {
                double sn, cs;
                sincos_turns_quad(s64_turns_to_f64(xhi[z]), sn, cs);
                add_rotations16(cs * a[z], sn * a[z], rc[z], rs[z], v);
                const uint64_t nlo = xlo[z] + dlo[z];
                xhi[z] = xhi[z] + dhi[z] + (nlo < xlo[z] ? 1 : 0);
                xlo[z] = nlo;
            }
#pragma unroll
            for (int i = 0; i < HIT_MB; ++i)
                for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < HIT_MB; ++i)
                    if (mb + i < n_m) acc[warp * n_m + mb + i] += v[i];
            }
        }
    }
    __syncthreads();
    for (int m = threadIdx.x; m < n_m; m += HIT_THREADS) {
        double s = 0.0;
        for (int w = 0; w < HIT_THREADS / 32; ++w) s += acc[w * n_m + m];
        partial[(int64_t)blockIdx.x * n_m + m] = s;
    }
}

__global__ void hit_reduce_kernel(const double *partial, int64_t P, int n_split, int n_m, double *h) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= P * n_m) return;
    const int64_t p = idx / n_m;
    const int m = (int)(idx - p * n_m);
    double s = 0.0;
    for (int c = 0; c < n_split; ++c) s += partial[(p * n_split + c) * n_m + m];
    h[idx] = s;
}

__global__ void scan_reduce_kernel(const double *partial, int P, int n_chunk, int n_m, double *h) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)P * n_m) return;
    const int p = (int)(idx / n_m), m = (int)(idx - (int64_t)p * n_m);
    double s = 0.0;
    for (int c = 0; c < n_chunk; ++c) s += partial[((int64_t)p * n_chunk + c) * n_m + m];
    h[idx] = s;
}

// ------------------------------------------------------------------ scans on cell moments
//
// Each base point's grid is cut into NB blocks of Bp points; the moments about each block's middle
// point (64.64, exact) are taken once per zero and evaluated on the block's points (k2_cells.h).

typedef unsigned __int128 u128;

struct ScanPlan {
    int Bp = 0, NB = 0, d1 = 0;
    int64_t chunk = 0;         // base points per pass
    CellPlan cp;
};

constexpr size_t SCAN_MOMENT_BYTES = (size_t)256 << 20;
constexpr int64_t SCAN_MAX_POINTS = 65535;                  // block points per pass (a grid dimension)

// Chooses the block count and the series length with the smallest estimated work; false when the direct
// kernel is the cheaper one (c_old: its warp cycles per 32 (point, zero) pairs): few points per base,
// or a step so large that a block's cells hold less than a few zeros each.  The estimates are warp cycles
// of one scheduler, fitted to the kernels' measured times: a moment step (32 pairs) ~120 for the phasors + 20 per mma, the staging ~20 per zero and
// CTA, 32 points of the evaluation 3.6 per FP64 operation, 2 D1 + 15 of them per cell.
bool plan_scan(const Table &t, int64_t P, int64_t n_use, int64_t n_m, uint64_t step_int, uint64_t step_frac,
               double c_old, int64_t old_points, ScanPlan &best) {
    if (n_use < 1 || step_int >> 31) return false;
    const double step = (double)step_int + (double)step_frac * 0x1p-64;
    double best_cost = c_old / 32.0 * P * old_points * n_use;
    bool found = false;
    for (int64_t NB = 1; NB <= n_m; NB = NB < 64 ? 2 * NB : NB + 64) {
        const int64_t Bp = (n_m + NB - 1) / NB;
        if (NB > 1 && Bp < 32) break;
        if (NB > SCAN_MAX_POINTS) break;
        const int64_t pts = P * NB;
        for (int d1 : {8, 16}) {
            const int ppc = cell_peaks(pts, d1);
            const double tiles = (double)((pts + ppc - 1) / ppc);
            // at least one item per CTA slot where the cells hold 16 zeros or more
            const int64_t min_cells = std::min<int64_t>(n_use / 16, (int64_t)(296 / tiles));
            CellPlan cp;
            if (!plan_cells(t, n_use, 0, (double)((Bp + 1) / 2) * step, d1, min_cells, cp)) continue;
            const double nc = cp.cells();
            const double zeros = n_use + 2.0 * nc;
            // one moment item per SM keeps it busy; however few they are, a scan CTA (256 points) takes the
            // latency of its cells, three CTAs to an SM
            const double mom = tiles * zeros * (ppc / 32.0 * (120.0 + 5.0 * d1) + 20.0) / std::min(1.0, nc * tiles / 148.0);
            const double ctas = (double)pts * cell_scan_ctas(Bp);
            const double eval = nc * (2 * d1 + 15) * std::max(ctas * 8.0 * 1.8, 592.0 * 4.0 * std::ceil(ctas / 444.0));
            const double bytes = (double)NB * nc * 2 * d1 * 8;
            if (bytes > (double)SCAN_MOMENT_BYTES) continue;
            if (mom + eval < best_cost) {
                best_cost = mom + eval;
                best.Bp = (int)Bp;
                best.NB = (int)NB;
                best.d1 = d1;
                best.cp = cp;
                best.chunk = std::max<int64_t>(
                    1, std::min({P, SCAN_MAX_POINTS / NB, (int64_t)((double)SCAN_MOMENT_BYTES / bytes)}));
                found = true;
            }
        }
    }
    return found;
}

// Whether v + m step stays in [0, 2^64) for m0 <= m <= m0 + n_m (the blocks' span) at every base point, so
// that each block's middle point is a 64.64 number.
bool scan_in_range(int64_t P, const uint64_t *vi, const uint64_t *vf, u128 step, int64_t m0, int64_t n_m) {
    const u128 lo = step * (u128)(m0 < 0 ? -m0 : 0), hi = step * (u128)std::max<int64_t>(0, m0 + n_m);
    for (int64_t p = 0; p < P; ++p) {
        const u128 v = (u128)vi[p] << 64 | vf[p];
        if (v < lo || v + hi < v) return false;
    }
    return true;
}

// The scan of P base points on cell moments (NO_ROOM, with nothing queued, where the device has no room for
// them); take(p0, np, d_h) queues what is done with the results of the
// base points [p0, p0 + np) (device, np x n_m) on t.stream.
template <typename Take>
int scan_cells(Table &t, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k, uint64_t step_int,
               uint64_t step_frac, int64_t m0, int64_t n_m, const ScanPlan &sp, Take take) {
    const u128 step = (u128)step_int << 64 | step_frac;
    const int64_t per = sp.chunk * sp.NB;
    const size_t pb = (size_t)per * 8, cb = cells_bytes(sp.cp);
    bool room;
    MB_TRY(t.io.ensure(2 * (pb + 256) + cb + 256 + (size_t)sp.chunk * n_m * 8 + 256, &room));
    if (room) MB_TRY(t.moments.ensure((size_t)per * sp.cp.cells() * 2 * sp.d1 * 8, &room));
    if (!room) return NO_ROOM;
    char *q = (char *)t.io.p;
    uint64_t *d_v = carve<uint64_t>(q, 2 * per);
    void *cbuf = carve<char>(q, cb);
    double *d_h = carve<double>(q, sp.chunk * n_m);
    double *M = (double *)t.moments.p;
    Cells cells;
    MB_TRY(build_cells(t, sp.cp, cbuf, cells, t.stream));
    std::vector<uint64_t> pts(2 * per);
    for (int64_t p0 = 0; p0 < P; p0 += sp.chunk) {
        const int64_t np = std::min(sp.chunk, P - p0), nb = np * sp.NB;
        for (int64_t p = 0; p < np; ++p)
            for (int64_t b = 0; b < sp.NB; ++b) {
                const int64_t m = m0 + b * sp.Bp + sp.Bp / 2;
                const u128 off = step * (u128)(m < 0 ? -m : m);
                const u128 v = (u128)v_int[p0 + p] << 64 | v_frac[p0 + p];
                const u128 y = m < 0 ? v - off : v + off;
                pts[p * sp.NB + b] = (uint64_t)(y >> 64);
                pts[nb + p * sp.NB + b] = (uint64_t)y;
            }
        MB_CUDA(cudaMemcpyAsync(d_v, pts.data(), 2 * (size_t)nb * 8, cudaMemcpyHostToDevice, t.stream));
        MB_TRY(launch_moments_gauss(t, cells, d_v, d_v + nb, nb, k, sp.d1, M, t.stream));
        MB_TRY(launch_cell_scan(t, cells, sp.d1, M, np, sp.NB, sp.Bp, n_m, step_int, step_frac, d_h, t.stream));
        MB_TRY(take(p0, np, (const double *)d_h));
    }
    return MB_OK;
}

// The first point of largest |h| of each base point's grid; a NaN ranks above every number (numpy.argmax).
struct HitBest {
    double h;
    int64_t m;
};
__global__ void __launch_bounds__(128) hit_best_kernel(const double *h, int n_m, HitBest *best) {
    __shared__ long long sv[4];
    __shared__ int si[4];
    const double *row = h + (int64_t)blockIdx.x * n_m;
    // |h| as its bits: ordered as the values are, one NaN above infinity
    auto key = [](double x) { return x != x ? 0x7ff8000000000000ll : __double_as_longlong(fabs(x)); };
    long long bv = -1;
    int bi = n_m;
    for (int m = threadIdx.x; m < n_m; m += 128) {
        const long long v = key(row[m]);
        if (v > bv) {
            bv = v;
            bi = m;
        }
    }
    auto take = [&](long long v, int i) {
        if (v > bv || (v == bv && i < bi)) {
            bv = v;
            bi = i;
        }
    };
    for (int o = 16; o > 0; o >>= 1) {
        const long long v = __shfl_xor_sync(0xffffffffu, bv, o);
        take(v, __shfl_xor_sync(0xffffffffu, bi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sv[threadIdx.x >> 5] = bv;
        si[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 4; ++w) take(sv[w], si[w]);
        best[blockIdx.x] = HitBest{row[bi], bi};
    }
}

// Warp cycles of the direct kernels per 32 (point, zero) pairs, from their measured times (25,001 points x
// 98,624 zeros in 1.36 ms; 256 x 241 points x 600,000 zeros in 33.6 ms).
constexpr double GRID_CYCLES = 20.0, HIT_CYCLES = 34.0;

}  // namespace
}  // namespace mb

using namespace mb;

// Copies a scan's results to the host.
struct ToHost {
    double *out;
    int64_t n_m;
    cudaStream_t s;
    int operator()(int64_t p0, int64_t np, const double *d_h) const {
        MB_CUDA(cudaMemcpyAsync(out + p0 * n_m, d_h, (size_t)np * n_m * 8, cudaMemcpyDeviceToHost, s));
        return MB_OK;
    }
};

extern "C" int mb_grid_scan(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k,
                            double T, uint64_t step_int, uint64_t step_frac, int64_t m0, int64_t n_m, double *out_h) {
    MB_CHECK_ARG(h && v_int && v_frac && out_h, "mb_grid_scan: null argument");
    MB_CHECK_ARG(P >= 0 && P <= 65535, "mb_grid_scan: P=%lld (0..65535)", (long long)P);
    MB_CHECK_ARG(n_m >= 0 && n_m <= (1 << 26) && P * n_m <= ((int64_t)1 << 28), "mb_grid_scan: n_m=%lld", (long long)n_m);
    MB_CHECK_ARG(m0 > -((int64_t)1 << 31) && m0 + n_m < ((int64_t)1 << 31), "mb_grid_scan: grid indices exceed 2^31");
    MB_CHECK_ARG(std::isfinite(k) && k >= 0.0 && !std::isnan(T), "mb_grid_scan: bad k or T");
    if (P == 0 || n_m == 0) return MB_OK;
    Table &t = table_of(h);
    MB_TRY(device_guard(t.device));
    const int64_t n_use = t.count_below(T);
    ScanPlan sp;
    const int64_t grid_points = (n_m + SCAN_THREADS * SCAN_MPT - 1) / (SCAN_THREADS * SCAN_MPT) * (SCAN_THREADS * SCAN_MPT);
    if (plan_scan(t, P, n_use, n_m, step_int, step_frac, GRID_CYCLES, grid_points, sp) &&
        scan_in_range(P, v_int, v_frac, (u128)step_int << 64 | step_frac, m0, (int64_t)sp.NB * sp.Bp))
    {
        const int st = scan_cells(t, P, v_int, v_frac, k, step_int, step_frac, m0, n_m, sp, ToHost{out_h, n_m, t.stream});
        if (st != MB_OK && st != NO_ROOM) return st;
        if (st == MB_OK) {
            MB_CUDA(cudaStreamSynchronize(t.stream));
            return MB_OK;
        }
    }
    const size_t cb = (size_t)P * 8, hb = (size_t)P * n_m * 8;
    int sms = 148;
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t.device));
    const int64_t per_cta = (int64_t)SCAN_THREADS * SCAN_MPT;
    const int64_t n_mt = (n_m + per_cta - 1) / per_cta;
    int64_t n_chunk = std::max<int64_t>(1, ((int64_t)sms * 4 + n_mt * P - 1) / (n_mt * P));
    n_chunk = std::min<int64_t>(n_chunk, std::max<int64_t>(1, (n_use + SCAN_TILE - 1) / SCAN_TILE));
    int64_t chunk = std::max<int64_t>(SCAN_TILE, ((n_use + n_chunk - 1) / n_chunk + SCAN_TILE - 1) / SCAN_TILE * SCAN_TILE);
    n_chunk = std::max<int64_t>(1, (n_use + chunk - 1) / chunk);
    MB_TRY(t.io.ensure(2 * cb + hb + 256));
    MB_TRY(t.work.ensure((size_t)P * n_chunk * n_m * 8));
    char *base = (char *)t.io.p;
    uint64_t *d_vi = (uint64_t *)base, *d_vf = (uint64_t *)(base + cb);
    double *d_h = (double *)(base + ((2 * cb + 255) & ~(size_t)255));
    double *partial = (double *)t.work.p;
    MB_CUDA(cudaMemcpyAsync(d_vi, v_int, cb, cudaMemcpyHostToDevice, t.stream));
    MB_CUDA(cudaMemcpyAsync(d_vf, v_frac, cb, cudaMemcpyHostToDevice, t.stream));
    if (n_use == 0) {
        MB_CUDA(cudaMemsetAsync(partial, 0, (size_t)P * n_m * 8, t.stream));
        n_chunk = 1;
    } else {
        dim3 grid((unsigned)n_mt, (unsigned)n_chunk, (unsigned)P);
        k2_scan_kernel<<<grid, SCAN_THREADS, 0, t.stream>>>(view(t), d_vi, d_vf, step_int, step_frac, m0, (int)n_m,
                                                            n_use, chunk, k, partial);
        MB_CUDA(cudaGetLastError());
    }
    const int64_t total = P * n_m;
    scan_reduce_kernel<<<(unsigned)((total + 255) / 256), 256, 0, t.stream>>>(partial, (int)P, (int)n_chunk, (int)n_m, d_h);
    MB_CUDA(cudaGetLastError());
    MB_CUDA(cudaMemcpyAsync(out_h, d_h, hb, cudaMemcpyDeviceToHost, t.stream));
    MB_CUDA(cudaStreamSynchronize(t.stream));
    return MB_OK;
}

// The scan of mb_hit_scan by whichever way is the cheaper, its results handed to take (see scan_cells).
template <typename Take>
static int hit_scan(Table &t, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k, int64_t n_use,
                    uint64_t step_int, uint64_t step_frac, int64_t m0, int64_t n_m, Take take) {
    ScanPlan sp;
    if (plan_scan(t, P, n_use, n_m, step_int, step_frac, HIT_CYCLES, (n_m + HIT_MB - 1) / HIT_MB * HIT_MB, sp) &&
        scan_in_range(P, v_int, v_frac, (u128)step_int << 64 | step_frac, m0, (int64_t)sp.NB * sp.Bp)) {
        const int st = scan_cells(t, P, v_int, v_frac, k, step_int, step_frac, m0, n_m, sp, take);
        if (st != NO_ROOM) return st;
    }
    const size_t cb = (size_t)P * 8, hb = (size_t)P * n_m * 8;
    MB_TRY(t.io.ensure(2 * cb + hb + 256));
    char *base = (char *)t.io.p;
    uint64_t *d_vi = (uint64_t *)base, *d_vf = (uint64_t *)(base + cb);
    double *d_h = (double *)(base + ((2 * cb + 255) & ~(size_t)255));
    MB_CUDA(cudaMemcpyAsync(d_vi, v_int, cb, cudaMemcpyHostToDevice, t.stream));
    MB_CUDA(cudaMemcpyAsync(d_vf, v_frac, cb, cudaMemcpyHostToDevice, t.stream));
    // splits per hit: about 8 CTAs per SM in all, each split at least two rounds of zeros
    int sms = 148;
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t.device));
    const int64_t rounds = (n_use + HIT_THREADS * HIT_ZPT - 1) / (HIT_THREADS * HIT_ZPT);
    const int n_split = (int)std::max<int64_t>(1, std::min<int64_t>((8 * sms + P - 1) / P, rounds / 2));
    MB_TRY(t.work.ensure((size_t)P * n_split * n_m * sizeof(double)));
    double *partial = (double *)t.work.p;
    const size_t smem = (size_t)(HIT_THREADS / 32) * n_m * sizeof(double);
    if (smem > 48 * 1024)
        MB_CUDA(cudaFuncSetAttribute(k2_hit_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k2_hit_scan_kernel<<<(unsigned)(P * n_split), HIT_THREADS, smem, t.stream>>>(
        view(t), d_vi, d_vf, step_int, step_frac, m0, (int)n_m, n_use, k, n_split, partial);
    MB_CUDA(cudaGetLastError());
    hit_reduce_kernel<<<(unsigned)((P * n_m + 255) / 256), 256, 0, t.stream>>>(partial, P, n_split, (int)n_m, d_h);
    MB_CUDA(cudaGetLastError());
    return take((int64_t)0, P, (const double *)d_h);
}

extern "C" int mb_hit_scan(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k,
                           int64_t n_use, uint64_t step_int, uint64_t step_frac, int64_t m0, int64_t n_m,
                           double *out_h) {
    MB_CHECK_ARG(h && v_int && v_frac && out_h, "mb_hit_scan: null argument");
    MB_CHECK_ARG(P >= 0 && P <= (1 << 24), "mb_hit_scan: P=%lld", (long long)P);
    MB_CHECK_ARG(n_m >= 1 && n_m <= HIT_MAX_M, "mb_hit_scan: n_m=%lld (1..%d)", (long long)n_m, HIT_MAX_M);
    MB_CHECK_ARG(m0 > -((int64_t)1 << 31) && m0 + n_m < ((int64_t)1 << 31), "mb_hit_scan: grid indices exceed 2^31");
    MB_CHECK_ARG(std::isfinite(k) && k >= 0.0, "mb_hit_scan: k=%g", k);
    if (P == 0) return MB_OK;
    Table &t = table_of(h);
    MB_CHECK_ARG(n_use >= 0 && n_use <= t.n, "mb_hit_scan: n_use=%lld of %lld", (long long)n_use, (long long)t.n);
    MB_TRY(device_guard(t.device));
    MB_TRY(hit_scan(t, P, v_int, v_frac, k, n_use, step_int, step_frac, m0, n_m, ToHost{out_h, n_m, t.stream}));
    MB_CUDA(cudaStreamSynchronize(t.stream));
    return MB_OK;
}

extern "C" int mb_hit_polish(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k,
                             int n_stages, const int64_t *zeros, const int64_t *m_half, const uint64_t *steps,
                             const int *recentre, const int *keep_h, const double *threshold, double *out_h,
                             double *out_dy, int64_t *out_stage) {
    const char *who = "mb_hit_polish";
    MB_CHECK_ARG(h && zeros && m_half && steps && recentre && keep_h && threshold, "%s: null argument", who);
    MB_CHECK_ARG(P >= 0 && P <= (1 << 24), "%s: P=%lld", who, (long long)P);
    MB_CHECK_ARG(n_stages >= 1 && n_stages <= 64, "%s: n_stages=%d", who, n_stages);
    MB_CHECK_ARG(std::isfinite(k) && k >= 0.0, "%s: k=%g", who, k);
    Table &t = table_of(h);
    for (int s = 0; s < n_stages; ++s)
        MB_CHECK_ARG(zeros[s] >= 0 && m_half[s] >= 0 && 2 * m_half[s] + 1 <= HIT_MAX_M, "%s: stage %d", who, s);
    if (P == 0) return MB_OK;
    MB_CHECK_ARG(v_int && v_frac && out_h && out_dy && out_stage, "%s: null array", who);
    MB_TRY(device_guard(t.device));
    typedef __int128 i128;
    std::vector<i128> centre(P, 0);
    std::vector<int64_t> alive(P);
    for (int64_t p = 0; p < P; ++p) {
        alive[p] = p;
        out_h[p] = out_dy[p] = 0.0;
        out_stage[p] = 0;
    }
    std::vector<uint64_t> vi(P), vf(P);
    std::vector<HitBest> best(P);
    MB_TRY(t.redo.ensure((size_t)P * sizeof(HitBest)));
    HitBest *d_best = (HitBest *)t.redo.p;
    for (int s = 0; s < n_stages && !alive.empty(); ++s) {
        const int64_t na = (int64_t)alive.size(), n_m = 2 * m_half[s] + 1;
        for (int64_t i = 0; i < na; ++i) {
            u128 v = (u128)v_int[alive[i]] << 64 | v_frac[alive[i]];
            if (recentre[s]) v += (u128)centre[alive[i]];
            vi[i] = (uint64_t)(v >> 64);
            vf[i] = (uint64_t)v;
        }
        auto take = [&](int64_t p0, int64_t np, const double *d_h) {
            hit_best_kernel<<<(unsigned)np, 128, 0, t.stream>>>(d_h, (int)n_m, d_best + p0);
            MB_CUDA(cudaGetLastError());
            return MB_OK;
        };
        MB_TRY(hit_scan(t, na, vi.data(), vf.data(), k, std::min(zeros[s], t.n), steps[2 * s], steps[2 * s + 1],
                        -m_half[s], n_m, take));
        MB_CUDA(cudaMemcpyAsync(best.data(), d_best, (size_t)na * sizeof(HitBest), cudaMemcpyDeviceToHost, t.stream));
        MB_CUDA(cudaStreamSynchronize(t.stream));
        const i128 step = (i128)((u128)steps[2 * s] << 64 | steps[2 * s + 1]);
        int64_t kept = 0;
        for (int64_t i = 0; i < na; ++i) {
            const int64_t p = alive[i];
            const i128 c = (recentre[s] ? centre[p] : 0) + (i128)(best[i].m - m_half[s]) * step;
            out_stage[p] = s;
            if (keep_h[s]) out_h[p] = best[i].h;
            centre[p] = c;
            out_dy[p] = (double)c * 0x1p-64;
            if (threshold[s] == -INFINITY || std::fabs(best[i].h) >= threshold[s]) alive[kept++] = p;
        }
        alive.resize(kept);
    }
    return MB_OK;
}
