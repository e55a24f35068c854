// Cell moments (see k2_cells.h), their evaluation on offset grids and the polishes on them.
//
// The moment pass is a contraction: for each cell, [peaks x zeros] unit phasors times [zeros x
// columns] weighted powers.  It runs on the FP64 tensor instruction (mma.m8n8k4.f64).  That
// instruction's A fragment holds one (row, k) element per lane, so with rows = 8 peaks and k = 4
// zeros each lane computes the exact phase and the (cos, sin) of its own (peak, zero) pair in
// registers -- the cosine is its A element of the real product, the sine that of the imaginary
// product -- and no phasor is ever stored.  The powers (B) come from shared memory, staged once per
// tile of zeros for the CTA's 64 or 128 peaks.
#include <algorithm>
#include <cmath>

#include <cuda_pipeline.h>

#include "k2_cells.h"
#include "k2_common.cuh"
#include "k2_phasor.cuh"
#include "k2_polish.cuh"

namespace mb {
namespace {

constexpr int CELL_THREADS = 256;

// ------------------------------------------------------------------ phasors

MB_DEV uint64_t wide(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
MB_DEV uint64_t wide_add(uint32_t a, uint32_t b, uint64_t c) {
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// A zero for the phase in units of 2^-60 turn: the limbs of G 2^124 (G 2^128 shifted down four bits, so the
// phase's fraction is where phasor() wants it), and arg(c) / 2pi 2^60 + 2^51 (half a table step).
struct ZRec {                   // 32 B
    uint32_t g0, g1, g2, g3, g4, pad;
    uint64_t psi;
};
MB_DEV ZRec zrec(uint32_t g0, uint32_t g1, uint32_t g2, uint32_t g3, uint32_t g4, uint64_t psi) {
    ZRec r;
    r.g0 = __funnelshift_r(g0, g1, 4);
    r.g1 = __funnelshift_r(g1, g2, 4);
    r.g2 = __funnelshift_r(g2, g3, 4);
    r.g3 = __funnelshift_r(g3, g4, 4);
    r.g4 = g4 >> 4;
    r.pad = 0;
    r.psi = (psi >> 4) + (1ull << 51);
    return r;
}

// floor(frac(v G) 2^60) less at most 7 units of 2^-60 turn (4e-17 rad: the carries out of the columns below),
// plus psi: columns 4 and 5 of phase128_exact and the high halves of column 3.
MB_DEV uint64_t phase60(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, const ZRec &z) {
    const uint64_t h3 = (wide(v0, z.g3) >> 32) + (wide(v1, z.g2) >> 32) + (wide(v2, z.g1) >> 32) + (wide(v3, z.g0) >> 32);
    const uint32_t top = v1 * z.g4 + v2 * z.g3 + v3 * z.g2;
    uint64_t acc = wide_add(v0, z.g4, z.psi + h3);
    acc = wide_add(v1, z.g3, acc);
    acc = wide_add(v2, z.g2, acc);
    acc = wide_add(v3, z.g1, acc);
    return acc + ((uint64_t)top << 32);
}

MB_DEV void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// ------------------------------------------------------------------ cells

struct CellGroups {
    int64_t a[2], b[2], e0[2];
    int nc[2];
};

// One warp per cell edge: a 32-way search of the group's zeros (four or five loads deep instead of the ~20
// of a binary search: 17 -> 5 us on 600,000 zeros).  Edge i of a group ends its cell i - 1 and starts cell i.
__global__ void cells_kernel(TabView t, CellGroups g, int64_t half, int *j0, int *j1, int64_t *ctr) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int q = w <= g.nc[0] ? 0 : 1, i = q ? w - g.nc[0] - 1 : w;      // nc + 1 edges each
    if (i > g.nc[q] || (q && g.nc[1] == 0)) return;
    const int64_t edge = g.e0[q] + 2 * half * i;
    // the first zero of the group at or above the edge (G in units of 2^-16, rounded down)
    int64_t lo = g.a[q], hi = g.b[q];
    if (i == 0) hi = lo;
    else if (i == g.nc[q]) lo = hi;
    while (lo < hi) {
        // 32 probes split [lo, hi) in 33 parts: the zeros below the edge are a prefix of the probes
        const int64_t m = lo + (hi - lo) * (lane + 1) / 33;
        const bool below = m < hi && ((int64_t)t.g4[m] << 16 | t.g3[m] >> 16) < edge;
        const int n = __popc(__ballot_sync(0xffffffffu, below));
        const int64_t nlo = n == 0 ? lo : lo + (hi - lo) * n / 33 + 1;
        hi = n == 32 ? hi : lo + (hi - lo) * (n + 1) / 33;
        lo = nlo;
    }
    if (lane == 0) {
        const int c = q ? g.nc[0] + i : i;
        if (i < g.nc[q]) {
            j0[c] = (int)lo;
            ctr[c] = edge + half;
        }
        if (i > 0) j1[c - 1] = (int)lo;
    }
}

// n chunks of the zeros [0, n_zeros) as cells (the power sums need no centre).  Their lengths grow with
// the zeros (edges n_zeros (c / n)^1.5): the lowest zeros carry most of the sum, and short chunks there
// keep the rounding of the running sums down.
__global__ void chunks_kernel(int64_t n_zeros, int n, int *j0, int *j1) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    auto edge = [&](int i) {
        const double x = (double)i / n;
        return i == n ? (int)n_zeros : (int)((double)n_zeros * x * sqrt(x));
    };
    j0[c] = edge(c);
    j1[c] = edge(c + 1);
}

// ------------------------------------------------------------------ moments

enum CellKind : int { CELL_GAUSS = 0, CELL_WEIGHTS = 1, CELL_POWERS = 2 };

// Columns of the power matrix: W series of D1 terms (both products), or the Taylor polish's nine even
// powers (real product, two tiles) and eight odd powers (imaginary product, one tile).
template <int KIND, int W, int D1>
struct CellShape {
    static constexpr int cols = KIND == CELL_POWERS ? 24 : (W * D1 + 7) / 8 * 8;
    static constexpr int NT = cols / 8;
    static constexpr int NTR = KIND == CELL_POWERS ? 2 : NT;      // tiles of the real product
    static constexpr int I0 = KIND == CELL_POWERS ? 2 : 0;        // first tile of the imaginary one
    static constexpr int NTI = NT - I0;
    // row stride in doubles = 4 mod 8: the 4 x 8 B fragment's half warps touch 16 distinct banks
    static constexpr int S = cols + 4;
    // a tile is TILE zeros x PARTS threads: a weight vector's D1 columns each, or two or four column groups
    // (two with 128 zeros where that leaves shared memory for three CTAs: the zeros' weights are then formed
    // twice instead of four times, 642 -> 602 us at 256 peaks x 600,000 zeros)
    static constexpr int PARTS = KIND == CELL_WEIGHTS ? W : (KIND == CELL_GAUSS && D1 == 8 ? 2 : 4);
    static constexpr int TILE = KIND == CELL_WEIGHTS ? (W == 5 ? 48 : 64) : CELL_THREADS / PARTS;
    static_assert(TILE * PARTS <= CELL_THREADS, "one (zero, part) per thread");
    // peaks per lane: two halve the reads of a zero's record and columns (a 16-term grid scan call
    // 178 -> 167 us, a Taylor polish of 1,024 peaks 605 -> 577).  One where the accumulators leave no
    // registers (weights), and with 8 terms, where three CTAs to an SM gain more (614 us, two peaks 630)
    static constexpr int MP = KIND == CELL_WEIGHTS || D1 == 8 ? 1 : 2;
    static constexpr int peaks = 64 * MP;                            // of one CTA
    static constexpr int ctas = MP == 1 && KIND != CELL_WEIGHTS ? 3 : 2;             // resident per SM
    static constexpr int smem = PH_BYTES + 2 * TILE * ((int)sizeof(ZRec) + S * 8);
    static constexpr int frag = 2 * (NTR + NTI);                   // accumulators per lane
};

// gamma - 2 pi G (at most 4 ulp of gamma): G's leading 53 bits and the rest times 2 pi in two parts, so the
// error is about 2^-100 G.
MB_DEV double gamma_excess(double gamma, uint32_t g4, uint32_t g3, uint32_t g2, uint32_t g1) {
    constexpr double P_HI = 6.283185307179586, P_LO = 2.4492935982947064e-16;       // 2 pi
    double h, l;
    two_sum(u32_to_f64(g4), u32_to_f64(g3) * 0x1p-32, h, l);
    l += fma(u32_to_f64(g2), 0x1p-64, u32_to_f64(g1) * 0x1p-96);
    const double p = P_HI * h, pe = fma(P_HI, h, -p);
    return (gamma - p) - (pe + fma(P_HI, l, P_LO * h));
}

// One tile of an item: the zeros [tb, min(tb + TILE, jb)) of a cell for one group of peaks.
struct CellTile {
    int item, cell, pt;
    uint32_t tb, jb;
};

// One item = one cell x Sh::peaks / nzw peaks.  Warp w serves 8 MP peaks from 8 MP (w / nzw) and the
// 4-zero steps congruent to w mod nzw; with nzw > 1 the warps' sums are added in warp order.
// Bound: instruction issue and the FP64 pipe together: an mma is 256 FMAs, 16 cycles of a scheduler's FP64 lanes, 2 of
// them per step and 8 columns, beside the phasor's 60 instructions, and little of the one hides the other (256
// points x 600,000 zeros with 8 terms: 620 us, where the FP64 operations alone need 290).  The next tile's zeros are loaded before the current one is summed and
// staged after it, into the other half of a double buffer, across items too: one barrier per tile.
template <int KIND, int W, int D1>
__global__ void __launch_bounds__(CELL_THREADS, (CellShape<KIND, W, D1>::ctas))
cell_moments_kernel(TabView t, const uint64_t *vi, const uint64_t *vf, const double *delta, const int *sel, int64_t P,
                    Cells cells, CellWeights wts, double k, int n_pt, int nzw, int n_items, double *out) {
    using Sh = CellShape<KIND, W, D1>;
    constexpr int TILE = Sh::TILE;
    extern __shared__ __align__(16) unsigned char smem[];
    double2 *tab = reinterpret_cast<double2 *>(smem);
    ZRec *rec_ = reinterpret_cast<ZRec *>(smem + PH_BYTES);                          // [2][TILE]
    double *E_ = reinterpret_cast<double *>(smem + PH_BYTES + 2 * TILE * sizeof(ZRec));   // [2][TILE][S]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cg = warp / nzw, zw = warp - cg * nzw;
    constexpr int MP = Sh::MP;
    const int ppc = Sh::peaks / nzw;
    const double inv_h = 1.0 / ((double)cells.half * 65536.0);     // units of 2^-32
    const double inv_kappa = 65536.0 / (6.283185307179586 * (double)cells.half);
    // this thread's part of a tile: zero sz, weight vector or column group sq
    const int sq = threadIdx.x / TILE, sz = threadIdx.x - sq * TILE;
    const double2 *copy = tab + (lane & (PH_COPIES - 1));
    const double *sw = wts.w[0];
    if constexpr (KIND == CELL_WEIGHTS) {
#pragma unroll
        for (int i = 1; i < W; ++i)
            if (sq == i) sw = wts.w[i];
    }
    auto open = [&](int item) {
        CellTile x;
        x.item = item;
        x.cell = item / n_pt;
        x.pt = item - x.cell * n_pt;
        x.tb = (uint32_t)cells.j0[x.cell];
        x.jb = (uint32_t)cells.j1[x.cell];
        return x;
    };
    // the zero's data in registers, then its record and columns into buffer b
    uint32_t g0, g1, g2, g3, g4;
    uint64_t psi;
    double al, gam, wv;
    auto fetch = [&](const CellTile &x) {
        const int nt = (int)(x.jb - x.tb);
        if (sq >= Sh::PARTS || sz >= min(TILE, (nt + 3) & ~3)) return;
        const int64_t j = (int64_t)x.tb + (sz < nt ? sz : 0);
        g1 = t.g1[j]; g2 = t.g2[j]; g3 = t.g3[j]; g4 = t.g4[j];
        if (sq == 0) {
            g0 = t.g0[j];
            psi = t.psi[j];
        }
        al = sz < nt ? 2.0 * t.alpha[j] : 0.0;
        gam = t.gamma[j];
        if constexpr (KIND != CELL_GAUSS) wv = sw[j];
    };
    auto stage = [&](const CellTile &x, int b) {
        const int nt = (int)(x.jb - x.tb);
        if (sq >= Sh::PARTS || sz >= min(TILE, (nt + 3) & ~3)) return;
        if (sq == 0) {
            rec_[b * TILE + sz] = zrec(g0, g1, g2, g3, g4, psi);
        }
        double *row = E_ + (b * TILE + sz) * Sh::S;
        if constexpr (KIND == CELL_POWERS) {
            const double u = gam * 1.0e-4, u2 = u * u, u4 = u2 * u2, u8 = u4 * u4;
            const double wa = al * wv;
            if (sq == 0) {                               // u^0 .. u^8
                double e = wa;
#pragma unroll
                for (int m = 0; m < 5; ++m, e *= u2) row[m] = e;
            } else if (sq == 1) {                        // u^10 .. u^16, then unused columns
                double e = wa * (u8 * u2);
#pragma unroll
                for (int m = 5; m < 9; ++m, e *= u2) row[m] = e;
#pragma unroll
                for (int m = 9; m < 16; ++m) row[m] = 0.0;
            } else {                                     // u^1 .. u^7, u^9 .. u^15
                double e = wa * (sq == 2 ? u : u8 * u);
#pragma unroll
                for (int m = 0; m < 4; ++m, e *= u2) row[16 + (sq - 2) * 4 + m] = e;
            }
        } else {
            const int64_t df = (int64_t)((uint64_t)g4 << 32 | g3) - (cells.ctr[x.cell] << 16);
            double y = ((double)df + u32_to_f64(g2) * 0x1p-32) * inv_h;
            // the polishes' offsets turn by the table's FP64 gamma, not 2 pi G
            if constexpr (KIND == CELL_WEIGHTS) y += gamma_excess(gam, g4, g3, g2, g1) * inv_kappa;
            if constexpr (KIND == CELL_GAUSS) {
                constexpr int C = D1 / Sh::PARTS;          // columns of a group, a power of two
                double step = y;                               // y^C
#pragma unroll
                for (int m = 1; m < C; m *= 2) step *= step;
                double e = al * exp(-k * gam * gam);
                if (sq & 1) e *= step;
                if (sq & 2) e *= step * step;
#pragma unroll
                for (int m = 0; m < C; ++m, e *= y) row[sq * C + m] = e;
            } else {
                double e = al * wv;
#pragma unroll
                for (int m = 0; m < D1; ++m, e *= y) row[sq * D1 + m] = e;
                if (sq == W - 1)
#pragma unroll
                    for (int m = W * D1; m < Sh::cols; ++m) row[m] = 0.0;
            }
        }
    };

    CellTile cur = open(blockIdx.x);                 // the grid is at most n_items CTAs
    fetch(cur);
    phasor_table_init(tab, CELL_THREADS);
    stage(cur, 0);
    __syncthreads();
    Cand64 v[MP];
    double aR[MP][Sh::NTR][2], aI[MP][Sh::NTI][2];
    bool first = true;
    for (int b = 0;; b ^= 1) {
        CellTile nxt = cur;
        nxt.tb += TILE;
        const bool last = nxt.tb >= cur.jb;          // the item's last tile (an empty cell has one)
        if (last) {
            nxt.item += gridDim.x;
            if (nxt.item < n_items) nxt = open(nxt.item);
        }
        const bool more = nxt.item < n_items;
        if (more) fetch(nxt);
        const int64_t pw = (int64_t)cur.pt * ppc + cg * 8 * MP;        // the warp's first peak
        const int64_t p0 = pw + (lane >> 2);                           // this lane's peaks: p0 + 8 m
        if (first) {
#pragma unroll
            for (int m = 0; m < MP; ++m) {
                v[m] = Cand64{0, 0};
                if (p0 + 8 * m < P) {
                    const int64_t i = sel ? sel[p0 + 8 * m] : p0 + 8 * m;
                    v[m] = fold_delta(vi[i], vf[i], delta ? delta[i] : 0.0);
                }
#pragma unroll
                for (int i = 0; i < Sh::NTR; ++i) aR[m][i][0] = aR[m][i][1] = 0.0;
#pragma unroll
                for (int i = 0; i < Sh::NTI; ++i) aI[m][i][0] = aI[m][i][1] = 0.0;
            }
        }
        if (pw < P) {
            const int n_step = (min(TILE, (int)(cur.jb - cur.tb)) + 3) >> 2;
            const ZRec *rp = rec_ + b * TILE + zw * 4 + (lane & 3);
            const double *bp = E_ + (b * TILE + zw * 4 + (lane & 3)) * Sh::S + (lane >> 2);
            const int dr = nzw * 4, de = dr * Sh::S;
#pragma unroll 2
            for (int st = zw; st < n_step; st += nzw, rp += dr, bp += de) {
                const ZRec z = *rp;
                double cs[MP], sn[MP];
#pragma unroll
                for (int m = 0; m < MP; ++m)
                    phasor(phase60((uint32_t)v[m].vf, (uint32_t)(v[m].vf >> 32), (uint32_t)v[m].vi,
                                   (uint32_t)(v[m].vi >> 32), z), copy, cs[m], sn[m]);
#pragma unroll
                for (int i = 0; i < Sh::NT; ++i) {
                    const double bv = bp[i * 8];
#pragma unroll
                    for (int m = 0; m < MP; ++m) {
                        if (i < Sh::NTR) dmma(aR[m][i], cs[m], bv);
                        if (i >= Sh::I0) dmma(aI[m][i - Sh::I0], sn[m], bv);
                    }
                }
            }
        }
        if (last) {
            if (nzw > 1) {                     // add the other warps' sums of this peak group, in order
                double *buf = E_ + cg * 32 * MP * Sh::frag;      // spans both halves of the tile buffer
                auto each = [&](auto f) {
#pragma unroll
                    for (int m = 0; m < MP; ++m) {
#pragma unroll
                        for (int i = 0; i < 2 * Sh::NTR; ++i) f(m * Sh::frag + i, aR[m][i >> 1][i & 1]);
#pragma unroll
                        for (int i = 0; i < 2 * Sh::NTI; ++i) f(m * Sh::frag + 2 * Sh::NTR + i, aI[m][i >> 1][i & 1]);
                    }
                };
                for (int w = 1; w < nzw; ++w) {
                    __syncthreads();
                    if (zw == w) each([&](int i, double &x) { buf[i * 32 + lane] = x; });
                    __syncthreads();
                    if (zw == 0) each([&](int i, double &x) { x += buf[i * 32 + lane]; });
                }
                __syncthreads();               // all read before the next tile is staged there
            }
            // C fragment: row = peak, columns 2 (lane mod 4) + {0, 1}
#pragma unroll
            for (int m = 0; m < MP; ++m) {
                const int64_t p = p0 + 8 * m;
                if (zw > 0 || p >= P) continue;
#pragma unroll
                for (int i = 0; i < Sh::NT; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int col = i * 8 + (lane & 3) * 2 + e;
                        if constexpr (KIND == CELL_POWERS) {
                            out[(p * cells.n + cur.cell) * 24 + col] = i < Sh::NTR ? aR[m][i < Sh::NTR ? i : 0][e]
                                                                                   : aI[m][i < Sh::NTR ? 0 : i - Sh::I0][e];
                        } else if (col < W * D1) {
                            const int w = col / D1, n = col - w * D1;
                            double *o = out + (((int64_t)w * P + p) * cells.n + cur.cell) * (2 * D1) + n;
                            o[0] = aR[m][i < Sh::NTR ? i : 0][e];
                            o[D1] = aI[m][i - Sh::I0 >= 0 ? i - Sh::I0 : 0][e];
                        }
                    }
            }
        }
        if (!more) break;
        stage(nxt, b ^ 1);
        __syncthreads();
        cur = nxt;
        first = last;
    }
}

int sm_count(const Table &t, int *sms) {
    MB_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, t.device));
    return MB_OK;
}

template <int KIND, int W, int D1>
int launch_moments(const Table &t, const Cells &c, const uint64_t *vi, const uint64_t *vf, const double *delta,
                   const int *sel, int64_t P, const CellWeights &w, double k, int nzw, double *out, cudaStream_t s) {
    using Sh = CellShape<KIND, W, D1>;
    static_assert(4 * 32 * Sh::MP * Sh::frag <= 2 * Sh::TILE * Sh::S || KIND == CELL_WEIGHTS, "reduction buffer");
    MB_TRY(cell_kernel_attributes());
    int sms = 148;
    MB_TRY(sm_count(t, &sms));
    const int64_t slots = (int64_t)Sh::ctas * sms;
    const int64_t n_pt = (P + Sh::peaks / nzw - 1) / (Sh::peaks / nzw);
    const int64_t items = n_pt * c.n;
    MB_CHECK_ARG(items < ((int64_t)1 << 31), "cell moments: %lld items", (long long)items);
    cell_moments_kernel<KIND, W, D1><<<(unsigned)std::min<int64_t>(slots, items), CELL_THREADS, Sh::smem, s>>>(
        view(t), vi, vf, delta, sel, P, c, w, k, (int)n_pt, nzw, (int)items, out);
    MB_CUDA(cudaGetLastError());
    return MB_OK;
}

// ------------------------------------------------------------------ offset scans

constexpr int CSCAN_CELLS = 32;                // cells staged at a time

// Thread: PT pairs of offsets +-m step of one block over every SPLIT-th cell.  The offset's sign changes
// only the signs of the odd terms and of the rotation's sine, so the pair costs one rotation and one series
// (256 x 241 points over 235 cells 60 -> 36 us; a scan call of 25,001 points 158 -> 143).  The moments are read
// as broadcasts.  With a few hundred CTAs the cells' dependent chains are exposed, hence the split (its sums are
// added in order) and the four products of each pair summed apart.  The next CSCAN_CELLS cells' moments are
// copied while the current ones are evaluated.
template <int D1, int SPLIT, int PT, int LANES>
__global__ void __launch_bounds__(LANES *SPLIT)
cell_scan_kernel(Cells cells, const double *M, int NB, int Bp, int64_t n_m, uint64_t si, uint64_t sf, double kstep,
                 double *out) {
    constexpr int THREADS = LANES * SPLIT;
    extern __shared__ __align__(16) unsigned char smem[];
    double2 *tab = reinterpret_cast<double2 *>(smem);
    double2 *mom_ = reinterpret_cast<double2 *>(smem + PH_BYTES);                 // [2][cell][D1]: pairs of one row
    ulonglong2 *dph_ = reinterpret_cast<ulonglong2 *>(mom_ + 2 * CSCAN_CELLS * D1);     // [2][cell] frac(step G_c): lo, hi
    const double2 *copy = tab + (threadIdx.x & (PH_COPIES - 1));
    phasor_table_init(tab, THREADS);
    const int part = threadIdx.x / LANES, tl = threadIdx.x - part * LANES;
    const int64_t pb = blockIdx.y;                               // point p NB + b
    const int64_t p = pb / NB, b = pb - p * NB;
    const int np = (int)min((int64_t)Bp, n_m - b * Bp);          // points of this block
    double e[PT][D1], h[PT][2];                      // h at +m and -m
    uint32_t ml[PT];
#pragma unroll
    for (int i = 0; i < PT; ++i) {
        ml[i] = (blockIdx.x * PT + i) * LANES + tl;
        // (kappa d)^n / n! with the sign of i^n: + + - -
        const double y = kstep * ml[i];
        double x = 1.0;
#pragma unroll
        for (int n = 0; n < D1; ++n) {
            e[i][n] = (n & 2) ? -x : x;
            x *= y * (1.0 / (n + 1));
        }
        h[i][0] = h[i][1] = 0.0;
    }
    // cells [cb, cb + CSCAN_CELLS): their moments on the way into half k of the buffer, this thread's centre
    auto fetch = [&](int cb, int k) -> int64_t {
        const int nc = min(CSCAN_CELLS, cells.n - cb);
        const double2 *src = reinterpret_cast<const double2 *>(M + (pb * cells.n + cb) * (2 * D1));
        for (int i = threadIdx.x; i < nc * D1; i += THREADS)
            __pipeline_memcpy_async(mom_ + k * CSCAN_CELLS * D1 + i, src + i, sizeof(double2));
        __pipeline_commit();
        return (int)threadIdx.x < nc ? cells.ctr[cb + threadIdx.x] : 0;
    };
    auto landed = [&](int64_t ctr, int k) {
        if (threadIdx.x < CSCAN_CELLS) {
            const uint64_t g = (uint64_t)ctr << 16;                                  // G_c 2^32
            uint64_t hi, lo;
            phase128_exact((uint32_t)sf, (uint32_t)(sf >> 32), (uint32_t)si, (uint32_t)(si >> 32), 0, 0, 0,
                           (uint32_t)g, (uint32_t)(g >> 32), hi, lo);
            dph_[k * CSCAN_CELLS + threadIdx.x] = make_ulonglong2(lo, hi);
        }
        __pipeline_wait_prior(0);
        __syncthreads();
    };
    if (cells.n > 0) landed(fetch(0, 0), 0);
    for (int cb = 0, k = 0; cb < cells.n; cb += CSCAN_CELLS, k ^= 1) {
        const int nc = min(CSCAN_CELLS, cells.n - cb);
        const bool more = cb + CSCAN_CELLS < cells.n;
        const int64_t ctr = more ? fetch(cb + CSCAN_CELLS, k ^ 1) : 0;
        const double2 *mom = mom_ + k * CSCAN_CELLS * D1;
        const ulonglong2 *dph = dph_ + k * CSCAN_CELLS;
        for (int c = part; c < nc; c += SPLIT) {
            const double2 *m2 = mom + c * D1;
            const ulonglong2 d = dph[c];
            double cs[PT], sn[PT];
#pragma unroll
            for (int i = 0; i < PT; ++i) {
                // frac(m step G_c) to 2^-64 turn
                const uint64_t w = wide(ml[i], (uint32_t)d.y) + ((uint64_t)(ml[i] * (uint32_t)(d.y >> 32)) << 32) +
                                   (wide(ml[i], (uint32_t)(d.x >> 32)) >> 32);
                phasor((w >> 4) + (1ull << 51), copy, cs[i], sn[i]);
            }
            double rr[PT], ri[PT], ir[PT], ii[PT];
#pragma unroll
            for (int i = 0; i < PT; ++i) rr[i] = ri[i] = ir[i] = ii[i] = 0.0;
#pragma unroll
            for (int n = 0; n < D1; n += 2) {
                const double2 re = m2[n / 2], im = m2[(D1 + n) / 2];
#pragma unroll
                for (int i = 0; i < PT; ++i) {
                    rr[i] = fma(e[i][n], re.x, rr[i]);
                    ri[i] = fma(e[i][n + 1], im.y, ri[i]);
                    ir[i] = fma(e[i][n], im.x, ir[i]);
                    ii[i] = fma(e[i][n + 1], re.y, ii[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < PT; ++i) {
                h[i][0] += fma(cs[i], rr[i] - ri[i], -sn[i] * (ir[i] + ii[i]));
                h[i][1] += fma(cs[i], rr[i] + ri[i], sn[i] * (ir[i] - ii[i]));
            }
        }
        if (more) landed(ctr, k ^ 1);
    }
    // the other parts' sums, in order (they take the moments' place)
    double *other = reinterpret_cast<double *>(mom_);
    for (int q = 1; q < SPLIT; ++q) {
        __syncthreads();
        if (part == q)
#pragma unroll
            for (int i = 0; i < 2 * PT; ++i) other[i * LANES + tl] = h[i >> 1][i & 1];
        __syncthreads();
        if (part == 0)
#pragma unroll
            for (int i = 0; i < 2 * PT; ++i) h[i >> 1][i & 1] += other[i * LANES + tl];
    }
    if (part > 0) return;
#pragma unroll
    for (int i = 0; i < PT; ++i) {
        const int l = Bp / 2 + (int)ml[i], r = Bp / 2 - (int)ml[i];
        if (l < np) out[p * n_m + b * Bp + l] = h[i][0];
        if (ml[i] > 0 && r >= 0 && r < np) out[p * n_m + b * Bp + r] = h[i][1];
    }
}

template <int D1>
constexpr int cscan_smem() {
    static_assert(2 * CSCAN_CELLS * D1 * 16 >= 2 * CSCAN_PAIRS * 8, "the parts' sums fit the moments' place");
    return PH_BYTES + 2 * CSCAN_CELLS * (D1 * 16 + 16);
}

// ------------------------------------------------------------------ polishes on moments

constexpr int CPOL_LD = 2 * CELL_D1 + 1;       // row of staged moments: an odd stride has no bank conflicts
__host__ __device__ constexpr int cpol_threads(bool staged) { return staged ? 512 : 256; }

// The part of a point's delta below 2^-64, which its fixed-point fold (fold_delta) dropped: at most 2^-65, an angle of
// up to 3.5e-14 at gamma = 1.3e6.
MB_DEV double delta_rest(double delta) {
    const double fixed = delta * 0x1p64;
    return (fixed - round(fixed)) * 0x1p-64;                     // ties away from zero, as fold_delta rounds
}

// The series at one offset: F0 = E Q0 and, with DERIV, F1 = E Q1, F2 = E Q2, where E = e^{2 pi i G_c d} and
// Q0 = sum M_n (i y)^n / n!, Q1, Q2 its first and second derivative in i y (y = kappa d).
// The rotation's offset is d + rho, rho = delta_rest of the point's delta (in the series it is far below rounding).
struct CellSeries {
    double d, rho, e[CELL_D1];
    MB_DEV CellSeries(double d_, double rho_, double kappa) : d(d_), rho(rho_) {
        const double y = kappa * d_;
        double x = 1.0;
#pragma unroll
        for (int n = 0; n < CELL_D1; ++n) {
            e[n] = (n & 2) ? -x : x;
            x *= y * (1.0 / (n + 1));
        }
    }
    // sum_{n >= s} M_n (i y)^{n - s} / (n - s)!
    template <int SHIFT>
    MB_DEV void q(const double *m, double &qr, double &qi) const {
        qr = qi = 0.0;
#pragma unroll
        for (int n = SHIFT; n < CELL_D1; ++n) {
            const double x = e[n - SHIFT], re = m[n], im = m[CELL_D1 + n];
            if ((n - SHIFT) & 1) {
                qr = fma(-x, im, qr);
                qi = fma(x, re, qi);
            } else {
                qr = fma(x, re, qr);
                qi = fma(x, im, qi);
            }
        }
    }
    // e^{2 pi i G (d + rho)}: the product's rounding error is carried into the angle
    MB_DEV void rot(double G, double &cs, double &sn) const {
        const double p = G * d, pe = fma(G, rho, fma(G, d, -p));
        sincospi(2.0 * ((p - rint(p)) + pe), &sn, &cs);
    }
};

// A peak for the second pass: its output, weight and point index, and Newton's starting offsets.
struct Redo {
    int64_t out;
    int w, point;
    double start[2];
};

template <int MODE>
struct PolishRule;              // Newton's constants and starts in each loop of k2_polish.cuh
template <>
struct PolishRule<POLISH_EVAL_FAST> {
    static constexpr int iters = 6, starts = 1;
    static constexpr double clamp = 1e-4, tol = 1e-13;
};
template <>
struct PolishRule<POLISH_SINGLE> {
    static constexpr int iters = 8, starts = 2;
    static constexpr double clamp = 2e-5, tol = 1e-14;
};
template <>
struct PolishRule<POLISH_TOPK> {
    static constexpr int iters = 4, starts = 1;
    static constexpr double clamp = 1e-5, tol = 1e-13;
};

// Whether a start's h replaces the best so far, in each loop's way.
template <int MODE>
MB_DEV bool polish_keep(double h, double best) {
    return MODE == POLISH_EVAL_FAST ? !(fabs(best) > fabs(h)) : fabs(h) > fabs(best);
}

// One CTA per (peak, weight vector).  STAGED: its moments in shared memory, read once and row by row.  From global
// memory every load of a warp touches 32 rows of 176 bytes, eight times over the Newton steps, and the kernel is
// bound by those wavefronts (1,280 polishes on 800 cells: 272 us, staged 206).
template <int MODE, bool STAGED>
__global__ void __launch_bounds__(cpol_threads(STAGED))
cell_polish_kernel(Cells cells, const double *M, CellPolishArgs a, const double *delta, Redo *redo, int *n_redo) {
    using R = PolishRule<MODE>;
    constexpr int THREADS = cpol_threads(STAGED), LD = STAGED ? CPOL_LD : 2 * CELL_D1;
    __shared__ double red[3][THREADS / 32];
    __shared__ double best_v[THREADS / 32];
    __shared__ int best_i[THREADS / 32];
    const int64_t p = blockIdx.x;
    const int w = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double *m0 = M + ((int64_t)w * a.P + p) * cells.n * (2 * CELL_D1);
    if constexpr (STAGED) {
        extern __shared__ double staged[];                       // [cell][CPOL_LD]
        for (int i = threadIdx.x; i < cells.n * (2 * CELL_D1); i += THREADS)
            __pipeline_memcpy_async(staged + i / (2 * CELL_D1) * CPOL_LD + i % (2 * CELL_D1), m0 + i, sizeof(double));
        __pipeline_commit();
        __pipeline_wait_prior(0);
        __syncthreads();
        m0 = staged;
    }
    const double H = (double)cells.half * 0x1p-16, kappa = 6.283185307179586 * H;
    const int64_t point = a.sel ? a.sel[p] : p;
    const int64_t o = (int64_t)w * a.out_stride + point;
    const double rho = delta ? delta_rest(delta[point]) : 0.0;

    // N sums over the CTA, every thread gets them (warp partials in warp order)
    auto block_sums = [&](auto &x) {
        constexpr int N = sizeof(x) / sizeof(double);
#pragma unroll
        for (int i = 0; i < N; ++i)
            for (int s = 16; s > 0; s >>= 1) x[i] += __shfl_xor_sync(0xffffffffu, x[i], s);
        __syncthreads();
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < N; ++i) red[i][warp] = x[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < N; ++i) {
            x[i] = 0.0;
#pragma unroll
            for (int s = 0; s < THREADS / 32; ++s) x[i] += red[i][s];
        }
    };
    auto value = [&](double d) {
        const CellSeries S(d, rho, kappa);
        double x[1] = {0.0};
        for (int c = threadIdx.x; c < cells.n; c += THREADS) {
            double cs, sn, qr, qi;
            S.rot((double)cells.ctr[c] * 0x1p-16, cs, sn);
            S.q<0>(m0 + c * LD, qr, qi);
            x[0] += cs * qr - sn * qi;
        }
        block_sums(x);
        return x[0];
    };
    // h(0); sqrt(sum gamma^4 |M_c0|^2): 2^-53 |d| times it is the size of the error that rounding
    // gamma_j d leaves in h'(d); and sum |Re M_c0| + |Im M_c0|, times POLISH_TIE the distance at which two |h| may be
    // told apart one way here and the other way by the loops over the zeros (shared: a register more spills)
    __shared__ double tie;
    double h0, noise;
    {
        double x[3] = {0.0, 0.0, 0.0};
        for (int c = threadIdx.x; c < cells.n; c += THREADS) {
            const double *m = m0 + c * LD;
            const double g = 6.283185307179586 * (double)cells.ctr[c] * 0x1p-16, g2 = g * g;
            x[0] += fma(-g * rho, m[CELL_D1], m[0]);             // the rotation by g rho to first order
            x[1] += g2 * g2 * (m[0] * m[0] + m[CELL_D1] * m[CELL_D1]);
            x[2] += fabs(m[0]) + fabs(m[CELL_D1]);
        }
        block_sums(x);
        h0 = x[0];
        noise = 0x1p-53 * sqrt(x[1]);
        if (threadIdx.x == 0) tie = POLISH_TIE * x[2];
    }
    // Newton on h' = 0 from d (the loop of polish_newton): with g = 2 pi G_c,
    //   h'  = -(g Im F0 + kappa Im F1),   h'' = -(g^2 Re F0 + 2 g kappa Re F1 + kappa^2 Re F2),
    // and for the sensitivity the third derivative's leading part.  A step d - h' / h'' multiplies the
    // error so far by |h' h3 / h''^2| and adds its own sums' error; a clamped step does neither.
    auto newton = [&](double d, double &sens) {
        sens = 0.0;
        for (int it = 0; it < R::iters; ++it) {
            const CellSeries S(d, rho, kappa);
            double x[3] = {0.0, 0.0, 0.0};
            for (int c = threadIdx.x; c < cells.n; c += THREADS) {
                const double *m = m0 + c * LD;
                const double G = (double)cells.ctr[c] * 0x1p-16, g = 6.283185307179586 * G;
                double cs, sn, q0r, q0i, q1r, q1i, q2r, q2i;
                S.rot(G, cs, sn);
                S.q<0>(m, q0r, q0i);
                S.q<1>(m, q1r, q1i);
                S.q<2>(m, q2r, q2i);
                const double ar = g * q0r + kappa * q1r, ai = g * q0i + kappa * q1i;
                const double br = g * (g * q0r + 2.0 * kappa * q1r) + kappa * kappa * q2r;
                const double bi = g * (g * q0i + 2.0 * kappa * q1i) + kappa * kappa * q2i;
                x[0] -= cs * ai + sn * ar;
                x[1] -= cs * br - sn * bi;
                x[2] += g * (cs * bi + sn * br);
            }
            block_sums(x);
            if (!(fabs(x[1]) > 1e-12)) break;
            double step = x[0] / x[1];
            if (fabs(step) < R::clamp)
                sens = sens * fabs(step * x[2] / x[1]) + noise * fmax(fabs(d), R::clamp) / fabs(x[1]);
            step = fmin(fmax(step, -R::clamp), R::clamp);
            d -= step;
            if (fabs(step) < R::tol) break;
        }
        return d;
    };
    // the first index in [0, n) of the largest |h(at(i))| over the cells [0, n_cells) if it exceeds `from`,
    // else -1: one warp per grid point
    auto grid_best = [&](int n, int n_cells, double from, auto at) {
        double bv = from;
        int bi = -1;
        for (int i = warp; i < n; i += THREADS / 32) {
            const CellSeries S(at(i), rho, kappa);
            double x = 0.0;
            for (int c = lane; c < n_cells; c += 32) {
                double cs, sn, qr, qi;
                S.rot((double)cells.ctr[c] * 0x1p-16, cs, sn);
                S.q<0>(m0 + c * LD, qr, qi);
                x += cs * qr - sn * qi;
            }
            for (int s = 16; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
            if (fabs(x) > bv) {
                bv = fabs(x);
                bi = i;
            }
        }
        __syncthreads();
        if (lane == 0) {
            best_v[warp] = bv;
            best_i[warp] = bi;
        }
        __syncthreads();
        bv = from;
        bi = -1;
        for (int s = 0; s < THREADS / 32; ++s)
            if (best_i[s] >= 0 && (best_v[s] > bv || (best_v[s] == bv && bi >= 0 && best_i[s] < bi))) {
                bv = best_v[s];
                bi = best_i[s];
            }
        return bi;
    };

    double hp = h0, dp = 0.0, start[2] = {0.0, 0.0};
    int ns = 1;
    if constexpr (MODE == POLISH_TOPK) {
        hp = h0 = a.h_unpol[o];                      // the grid stage's
        start[0] = a.ddy_pol[o];
    } else if constexpr (MODE == POLISH_EVAL_FAST) {
        const int steps = a.n_grid;
        auto at = [&](int i) { return (a.half * (i - steps)) / steps; };
        const int i = steps > 0 ? grid_best(2 * steps + 1, cells.n_first, fabs(h0), at) : -1;
        start[0] = i >= 0 ? at(i) : 0.0;
    } else if (a.n_grid > 0) {
        const int i = grid_best(a.n_grid, cells.n, -1.0, [&](int i) { return a.grid[i]; });
        start[1] = i >= 0 ? a.grid[i] : 0.0;
        ns = 2;
    }
    double worst = 0.0;
    for (int s = 0; s < ns; ++s) {
        double sens;
        const double d = newton(start[s], sens);
        const double h = value(d);
        if (!(sens <= worst)) worst = sens;
        if (fabs(fabs(h) - fabs(hp)) <= tie && fabs(d - dp) > R::tol) worst = INFINITY;
        if (polish_keep<MODE>(h, hp)) {
            hp = h;
            dp = d;
        }
    }
    if (threadIdx.x == 0) {
        a.h_unpol[o] = h0;
        a.h_pol[o] = hp;
        a.ddy_pol[o] = dp;
        if (!(worst <= POLISH_SENSITIVE * R::clamp)) redo[atomicAdd(n_redo, 1)] = Redo{o, w, (int)point, {start[0], start[1]}};
    }
}

// The second pass: the listed peaks' Newton and final value by the loops over the zeros, bit for bit as
// peak_polish_kernel forms them: POLISH_STRIDE running sums over zeros POLISH_STRIDE apart, warp trees, warps
// and CTA ranks in order.  One CTA per (32 of those sums, peak): eight warps form the terms of REDO_ROWS zeros
// of each sum at a time, a ninth adds the rows before in order.  Bound: instruction issue (an FP64 sincos
// per zero); with the terms written out by one kernel and added by a second one, a pass over seven peaks and
// 600,000 zeros took 33 + 31 us (memory traffic, then load latency), now 34.
constexpr int REDO_ROWS = 16, REDO_THREADS = 288, REDO_GROUPS = (int)(POLISH_STRIDE / 32);

struct RedoState {
    double d;
    int done, pad;
};

struct RedoBuf {
    const Redo *list;
    // A pass reads what the pass before wrote while other CTAs of its peak already write theirs, so both are
    // kept by the pass's parity.
    RedoState *state;           // [2][batch]
    double2 *slot;              // [2][batch][REDO_GROUPS]: the warp sums
    double *h_best, *d_best;    // [batch]
    double2 *ab;                // [batch][n]: (A, B)
    int batch;
};

__global__ void __launch_bounds__(256) redo_ab_kernel(ABExact src, int64_t n, RedoBuf rb) {
    const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (j >= n) return;
    double A, B;
    src.at(src.peak(rb.list[blockIdx.y].point), j, A, B);
    rb.ab[blockIdx.y * n + j] = make_double2(A, B);
}

MB_DEV double2 *redo_slots(const RedoBuf &rb, int it, int e) {
    return rb.slot + ((int64_t)(it & 1) * rb.batch + e) * REDO_GROUPS;
}

// The totals of pass `it`: a rank's warp sums in order (one lane each), then the ranks in order; every lane
// gets them.
MB_DEV double2 redo_total(const RedoBuf &rb, int it, int e) {
    constexpr int W = REDO_GROUPS / POLISH_CLUSTER;
    const double2 *slot = redo_slots(rb, it, e);
    const int rank = threadIdx.x & (POLISH_CLUSTER - 1);
    double2 x = make_double2(0.0, 0.0), t = x;
    for (int i = 0; i < W; ++i) {
        const double2 v = slot[rank * W + i];
        x.x += v.x;
        x.y += v.y;
    }
    for (int r = 0; r < POLISH_CLUSTER; ++r) {
        t.x += __shfl_sync(0xffffffffu, x.x, r);
        t.y += __shfl_sync(0xffffffffu, x.y, r);
    }
    return t;
}

// Pass `it` of a start's Newton loop; it == iters sums h itself.
template <int MODE>
__global__ void __launch_bounds__(REDO_THREADS, 4)
redo_pass_kernel(const double *gamma, int64_t n, CellWeights wts, RedoBuf rb, int start, int it) {
    using R = PolishRule<MODE>;
    constexpr int PER = REDO_ROWS / 8;                 // rows of one warp
    __shared__ double s_d[2][REDO_ROWS][32], s_dd[2][REDO_ROWS][32], s_w[2][REDO_ROWS][32];
    __shared__ RedoState s_state;
    const int e = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {                                   // the step of the pass before, alike in every CTA
        RedoState st;
        if (it == 0) {
            st = RedoState{rb.list[e].start[start], 0, 0};
        } else {
            st = rb.state[((it - 1) & 1) * rb.batch + e];
            const double2 t = redo_total(rb, it - 1, e);
            if (!st.done) {
                if (!(fabs(t.y) > 1e-12)) {
                    st.done = 1;
                } else {
                    double step = t.x / t.y;
                    step = fmin(fmax(step, -R::clamp), R::clamp);
                    st.d -= step;
                    if (fabs(step) < R::tol) st.done = 1;
                }
            }
        }
        if (lane == 0) {
            s_state = st;
            if (blockIdx.x == 0) rb.state[(it & 1) * rb.batch + e] = st;
        }
    }
    __syncthreads();
    const double d = s_state.d;
    const bool value = it == R::iters;
    if (s_state.done && !value) return;
    const double *w = wts.w[rb.list[e].w];
    const double2 *ab = rb.ab + (int64_t)e * n;
    const int64_t j0 = (int64_t)blockIdx.x * 32 + lane;             // this lane's sum: zeros j0 + i POLISH_STRIDE
    const int64_t first = n - (int64_t)blockIdx.x * 32;
    const int n_batch = first > 0 ? (int)((first + REDO_ROWS * POLISH_STRIDE - 1) / (REDO_ROWS * POLISH_STRIDE)) : 0;
    double2 v[PER];
    double g[PER], wv[PER], x = 0.0, y = 0.0;
    auto fetch = [&](int b) {                          // a row past the end adds 0
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int64_t j = j0 + ((int64_t)b * REDO_ROWS + warp * PER + i) * POLISH_STRIDE;
            const bool in = j < n;
            v[i] = in ? ab[j] : make_double2(0.0, 0.0);
            g[i] = in ? gamma[j] : 0.0;
            wv[i] = in ? w[j] : 0.0;
        }
    };
    if (warp < 8 && n_batch > 0) fetch(0);
    for (int b = 0; b <= n_batch; ++b) {
        if (warp < 8) {
            if (b < n_batch) {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    double sn, cs;
                    sincos(g[i] * d, &sn, &cs);
                    const double val = v[i].x * cs - v[i].y * sn;
                    const double dval = g[i] * (-v[i].x * sn - v[i].y * cs);
                    const int r = warp * PER + i;
                    s_d[b & 1][r][lane] = value ? val : dval;
                    s_dd[b & 1][r][lane] = -(g[i] * g[i]) * val;
                    s_w[b & 1][r][lane] = wv[i];
                }
                if (b + 1 < n_batch) fetch(b + 1);
            }
        } else if (b > 0) {
            const int c = (b - 1) & 1;
#pragma unroll
            for (int r = 0; r < REDO_ROWS; ++r) {
                const double u = s_w[c][r][lane];
                x += u * s_d[c][r][lane];
                if (!value) y += u * s_dd[c][r][lane];
            }
        }
        __syncthreads();
    }
    if (warp == 8) {
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, o);
            y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        if (lane == 0) redo_slots(rb, it, e)[blockIdx.x] = make_double2(x, y);
    }
}

// The start's h against the best so far; after the last start, the outputs.
template <int MODE>
__global__ void redo_keep_kernel(RedoBuf rb, CellPolishArgs a, int m, int start, bool last) {
    using R = PolishRule<MODE>;
    const int e = blockIdx.x;                          // a warp each
    if (e >= m) return;
    const int64_t o = rb.list[e].out;
    double hb = start == 0 ? a.h_unpol[o] : rb.h_best[e], db = start == 0 ? 0.0 : rb.d_best[e];
    const double h = redo_total(rb, R::iters, e).x;
    if (threadIdx.x > 0) return;
    if (polish_keep<MODE>(h, hb)) {
        hb = h;
        db = rb.state[(R::iters & 1) * rb.batch + e].d;
    }
    rb.h_best[e] = hb;
    rb.d_best[e] = db;
    if (last) {
        a.h_pol[o] = hb;
        a.ddy_pol[o] = db;
    }
}

// ------------------------------------------------------------------ Taylor polish, grid stage

constexpr int TAY_THREADS = 128;

// One CTA per peak: the chunks' power sums added in a fixed order (32 running sums over every 32nd chunk, then these
// pairwise: longer chains of sums near the total would round more than the loops over the zeros), then the grid
// points; ties of |h| go to the smaller index.
__global__ void __launch_bounds__(TAY_THREADS)
taylor_grid_kernel(const double *S, int n_chunk, const double *delta, const double *grid, int n_grid, double *h_unpol,
                   double *h_pol, double *ddy_pol) {
    __shared__ double part[4][24], mom[24];
    __shared__ double best_v[TAY_THREADS / 32], best_h[TAY_THREADS / 32];
    __shared__ int best_i[TAY_THREADS / 32];
    // (-1)^m/(2m)! and (-1)^m/(2m+1)!
    constexpr double CC[9] = {1.0, -1.0 / 2, 1.0 / 24, -1.0 / 720, 1.0 / 40320, -1.0 / 3628800,
                              1.0 / 479001600, -1.0 / 87178291200.0, 1.0 / 20922789888000.0};
    constexpr double CS[8] = {1.0, -1.0 / 6, 1.0 / 120, -1.0 / 5040, 1.0 / 362880, -1.0 / 39916800,
                              1.0 / 6227020800.0, -1.0 / 1307674368000.0};
    const int64_t p = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane < 24) {
        double x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = 0.0;
        const double *s = S + p * n_chunk * 24 + lane;
        int c = warp;
        for (; c + 28 < n_chunk; c += 32)
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] += s[(c + 4 * i) * 24];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + 4 * i < n_chunk) x[i] += s[(c + 4 * i) * 24];
        part[warp][lane] = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
    }
    __syncthreads();
    if (threadIdx.x < 24) mom[lane] = (part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]);
    __syncthreads();
    const double rho = delta ? delta_rest(delta[p]) : 0.0, h0 = fma(-rho * 1.0e4, mom[16], mom[0]);
    double bv = -1.0, hv = 0.0;
    int bi = n_grid;
    for (int g = threadIdx.x; g < n_grid; g += TAY_THREADS) {
        const double z = (grid[g] + rho) * 1.0e4, z2 = z * z;
        double hc = 0.0, hs = 0.0, pw = 1.0;
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            hc = fma(mom[m] * CC[m], pw, hc);
            if (m < 8) hs = fma(mom[16 + m] * CS[m], pw * z, hs);
            pw *= z2;
        }
        const double h = hc - hs;
        if (fabs(h) > bv) {
            bv = fabs(h);
            bi = g;
            hv = h;
        }
    }
    auto take = [&](double v2, int i2, double h2) {
        if (v2 > bv || (v2 == bv && i2 < bi)) {
            bv = v2;
            bi = i2;
            hv = h2;
        }
    };
    for (int o = 16; o > 0; o >>= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, bv, o), h2 = __shfl_xor_sync(0xffffffffu, hv, o);
        take(v2, __shfl_xor_sync(0xffffffffu, bi, o), h2);
    }
    if (lane == 0) {
        best_v[warp] = bv;
        best_i[warp] = bi;
        best_h[warp] = hv;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < TAY_THREADS / 32; ++w) take(best_v[w], best_i[w], best_h[w]);
        h_unpol[p] = h0;
        ddy_pol[p] = bi < n_grid ? grid[bi] : 0.0;
        h_pol[p] = bi < n_grid ? hv : h0;
    }
}

template <typename K>
int set_smem(K kern, int bytes) {
    MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared));
    return MB_OK;
}

}  // namespace

// Warps sharing a peak group's zeros in the scans: as many as keep the CTA's peak slots full,
// and two at least with 16 peaks a warp, unless there are peaks for eight full CTAs (fewer, larger items would
// not balance).
static int cell_nzw(int64_t P, int peaks) {
    int nzw = peaks == 128 && P < 8 * peaks ? 2 : 1;
    while (nzw < 8 && P <= peaks / (2 * nzw)) nzw *= 2;
    return nzw;
}

int cell_peaks(int64_t P, int d1) {
    const int peaks = d1 == 8 ? CellShape<CELL_GAUSS, 1, 8>::peaks : CellShape<CELL_GAUSS, 1, 16>::peaks;
    return peaks / cell_nzw(P, peaks);
}

int cell_kernel_attributes() {
    static void *done_ctx[64] = {};             // the context the attributes were set in
    int dev = 0;
    MB_CUDA(cudaGetDevice(&dev));
    void *ctx = current_context();
    if (dev >= 0 && dev < 64 && ctx && done_ctx[dev] == ctx) return MB_OK;
    MB_TRY(set_smem(cell_moments_kernel<CELL_GAUSS, 1, 8>, CellShape<CELL_GAUSS, 1, 8>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_GAUSS, 1, 16>, CellShape<CELL_GAUSS, 1, 16>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_WEIGHTS, 1, CELL_D1>, CellShape<CELL_WEIGHTS, 1, CELL_D1>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_WEIGHTS, 2, CELL_D1>, CellShape<CELL_WEIGHTS, 2, CELL_D1>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_WEIGHTS, 3, CELL_D1>, CellShape<CELL_WEIGHTS, 3, CELL_D1>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_WEIGHTS, 4, CELL_D1>, CellShape<CELL_WEIGHTS, 4, CELL_D1>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_WEIGHTS, 5, CELL_D1>, CellShape<CELL_WEIGHTS, 5, CELL_D1>::smem));
    MB_TRY(set_smem(cell_moments_kernel<CELL_POWERS, 1, 17>, CellShape<CELL_POWERS, 1, 17>::smem));
    MB_TRY(set_smem(cell_scan_kernel<8, 16, 1, 32>, cscan_smem<8>()));
    MB_TRY(set_smem(cell_scan_kernel<16, 16, 1, 32>, cscan_smem<16>()));
    MB_TRY(set_smem(cell_scan_kernel<8, 4, 2, 64>, cscan_smem<8>()));
    MB_TRY(set_smem(cell_scan_kernel<16, 4, 2, 64>, cscan_smem<16>()));
    MB_TRY(set_smem(cell_scan_kernel<8, 8, 2, 64>, cscan_smem<8>()));
    MB_TRY(set_smem(cell_scan_kernel<16, 8, 2, 64>, cscan_smem<16>()));
    if (dev >= 0 && dev < 64) done_ctx[dev] = current_context();
    return MB_OK;
}

bool plan_cells(const Table &t, int64_t n, int64_t split, double R, int d1, int64_t min_cells, CellPlan &out) {
    const double two_pi = 6.283185307179586;
    if (n < 1 || !(R >= 0.0) || !(t.h_gamma[n - 1] < two_pi * 0x1p30)) return false;
    // half width in units of 2^-16: 2 pi H R <= X
    const double want = R > 0.0 ? cell_x(d1) / (two_pi * R) * 65536.0 : 1e15;
    if (!(want >= 2.0)) return false;
    int64_t half = (int64_t)std::min(want, 1e12);
    const int64_t lo = (int64_t)std::floor(t.h_gamma[0] / two_pi * 65536.0) - 2;
    const int64_t hi = (int64_t)std::ceil(t.h_gamma[n - 1] / two_pi * 65536.0) + 2;
    // no wider than the zeros: with gamma far below the cells' centre, Newton's sums, formed about the centre,
    // would cancel
    half = std::min(half, std::max<int64_t>(2, (hi - lo + 1) / 2));
    if (min_cells > 1) half = std::min(half, std::max<int64_t>(2, (hi - lo) / (2 * min_cells)));
    out.half = half;
    auto group = [&](int q, int64_t a, int64_t b) {
        out.a[q] = a;
        out.b[q] = b;
        out.e0[q] = std::max<int64_t>(0, (int64_t)std::floor(t.h_gamma[a] / two_pi * 65536.0) - 2);
        const int64_t e1 = (int64_t)std::ceil(t.h_gamma[b - 1] / two_pi * 65536.0) + 2;
        const int64_t nc = (e1 - out.e0[q]) / (2 * half) + 1;
        out.nc[q] = (int)std::min<int64_t>(nc, (int64_t)1 << 30);
    };
    if (split > 0 && split < n) {
        out.groups = 2;
        group(0, 0, split);
        group(1, split, n);
    } else {
        out.groups = 1;
        group(0, 0, n);
        out.nc[1] = 0;
        out.a[1] = out.b[1] = out.e0[1] = 0;
    }
    return (int64_t)out.nc[0] + out.nc[1] < ((int64_t)1 << 28);
}

size_t cells_bytes(const CellPlan &p) { return ((size_t)p.cells() * 8 + 255) / 256 * 256 + 2 * (((size_t)p.cells() * 4 + 255) / 256 * 256); }

int build_cells(const Table &t, const CellPlan &p, void *buf, Cells &out, cudaStream_t s) {
    char *q = (char *)buf;
    const int n = p.cells();
    int64_t *ctr = carve<int64_t>(q, n);
    int *j0 = carve<int>(q, n), *j1 = carve<int>(q, n);
    CellGroups g;
    for (int i = 0; i < 2; ++i) {
        g.a[i] = p.a[i];
        g.b[i] = p.b[i];
        g.e0[i] = p.e0[i];
        g.nc[i] = p.nc[i];
    }
    cells_kernel<<<(unsigned)((n + 2 + 3) / 4), 128, 0, s>>>(view(t), g, p.half, j0, j1, ctr);
    MB_CUDA(cudaGetLastError());
    out = Cells{n, p.nc[0], p.half, j0, j1, ctr};
    return MB_OK;
}

int launch_moments_gauss(const Table &t, const Cells &c, const uint64_t *vi, const uint64_t *vf, int64_t P, double k,
                         int d1, double *out, cudaStream_t s) {
    const CellWeights none{};
    return d1 == 8 ? launch_moments<CELL_GAUSS, 1, 8>(t, c, vi, vf, nullptr, nullptr, P, none, k,
                                                      cell_nzw(P, CellShape<CELL_GAUSS, 1, 8>::peaks), out, s)
                   : launch_moments<CELL_GAUSS, 1, 16>(t, c, vi, vf, nullptr, nullptr, P, none, k,
                                                       cell_nzw(P, CellShape<CELL_GAUSS, 1, 16>::peaks), out, s);
}

int launch_moments_weights(const Table &t, const Cells &c, const uint64_t *vi, const uint64_t *vf,
                           const double *delta, const int *sel, int64_t P, int nw, const CellWeights &w,
                           double *out, cudaStream_t s) {
    // one warp per 8 peaks and zero order (nzw = 1) whatever P: a peak's moments keep their bits
    switch (nw) {
        case 1: return launch_moments<CELL_WEIGHTS, 1, CELL_D1>(t, c, vi, vf, delta, sel, P, w, 0.0, 1, out, s);
        case 2: return launch_moments<CELL_WEIGHTS, 2, CELL_D1>(t, c, vi, vf, delta, sel, P, w, 0.0, 1, out, s);
        case 3: return launch_moments<CELL_WEIGHTS, 3, CELL_D1>(t, c, vi, vf, delta, sel, P, w, 0.0, 1, out, s);
        case 4: return launch_moments<CELL_WEIGHTS, 4, CELL_D1>(t, c, vi, vf, delta, sel, P, w, 0.0, 1, out, s);
        default: return launch_moments<CELL_WEIGHTS, 5, CELL_D1>(t, c, vi, vf, delta, sel, P, w, 0.0, 1, out, s);
    }
}

// Chunks of 336 zeros on average, at most two per CTA slot, and one per SM where they hold 64 zeros.  Their number
// depends on the zeros alone and one warp adds a chunk's zeros, so a peak's sums keep their bits whatever the peaks
// beside it.  That costs calls of few peaks, whose CTAs have idle warps: one peak on 100,000 zeros 75 -> 88 us with
// eight warps to a chunk's zeros where there are 8 peaks, but two for all calls cost 1,024 peaks 490 -> 524.
int taylor_chunks(int64_t n) {
    return (int)std::max<int64_t>({1, std::min<int64_t>(592, n / 336), std::min<int64_t>(148, n / 64)});
}

size_t taylor_work_bytes(int64_t P, int n_chunk) {
    return 2 * ((size_t)n_chunk * 4 + 256) + (size_t)P * n_chunk * 24 * 8 + 256;
}

int launch_taylor_grid(const Table &t, const uint64_t *vi, const uint64_t *vf, const double *delta, int64_t P,
                       int64_t n, int n_chunk, const double *w, const double *grid, int n_grid, void *work,
                       double *h_unpol, double *h_pol, double *ddy_pol, cudaStream_t s) {
    char *q = (char *)work;
    int *j0 = carve<int>(q, n_chunk), *j1 = carve<int>(q, n_chunk);
    double *S = carve<double>(q, (size_t)P * n_chunk * 24);
    chunks_kernel<<<(unsigned)((n_chunk + 127) / 128), 128, 0, s>>>(n, n_chunk, j0, j1);
    MB_CUDA(cudaGetLastError());
    const Cells c{n_chunk, n_chunk, 1, j0, j1, nullptr};
    const CellWeights cw{{w}};
    MB_TRY((launch_moments<CELL_POWERS, 1, 17>(t, c, vi, vf, delta, nullptr, P, cw, 0.0, 1, S, s)));
    taylor_grid_kernel<<<(unsigned)P, TAY_THREADS, 0, s>>>(S, n_chunk, delta, grid, n_grid, h_unpol, h_pol, ddy_pol);
    MB_CUDA(cudaGetLastError());
    return MB_OK;
}

int launch_cell_scan(const Table &t, const Cells &c, int d1, const double *M, int64_t P, int NB, int Bp, int64_t n_m,
                     uint64_t step_int, uint64_t step_frac, double *out, cudaStream_t s) {
    MB_TRY(cell_kernel_attributes());
    const double step = (double)step_int + (double)step_frac * 0x1p-64;
    const double kstep = 6.283185307179586 * c.H() * step;
    int sms = 148;
    MB_TRY(sm_count(t, &sms));
    auto launch = [&](auto kernel, int pairs, int threads, int bytes) {
        const dim3 grid((unsigned)((Bp / 2 + pairs) / pairs), (unsigned)(P * NB));
        kernel<<<grid, threads, bytes, s>>>(c, M, NB, Bp, n_m, step_int, step_frac, kstep, out);
    };
    auto form = [&](auto few, auto one, auto many, int bytes) {
        const int64_t ctas = cell_scan_ctas(Bp) * P * NB;
        // a CTA per SM at most: the cells split eight ways (2 warps per scheduler otherwise); at most a quarter of
        // the SMs: 32 pairs a CTA instead of 128 (a scan of 801 points over 98,624 zeros 114 -> 93 us, 5,001: 119 -> 106)
        if (4 * ctas <= sms) launch(few, 32, 512, bytes);
        else if (ctas <= sms) launch(one, CSCAN_PAIRS, 512, bytes);
        else launch(many, CSCAN_PAIRS, 256, bytes);
    };
    if (d1 == 8)
        form(cell_scan_kernel<8, 16, 1, 32>, cell_scan_kernel<8, 8, 2, 64>, cell_scan_kernel<8, 4, 2, 64>, cscan_smem<8>());
    else
        form(cell_scan_kernel<16, 16, 1, 32>, cell_scan_kernel<16, 8, 2, 64>, cell_scan_kernel<16, 4, 2, 64>, cscan_smem<16>());
    MB_CUDA(cudaGetLastError());
    return MB_OK;
}

// Peaks of one batch of the second pass: their A and B take at most 256 MB.
static int redo_batch(int64_t count, int64_t n) {
    const int64_t fit = ((int64_t)256 << 20) / ((int64_t)sizeof(double2) * n);
    return (int)std::max<int64_t>(1, std::min<int64_t>({fit, count, 1024}));
}

size_t cell_polish_bytes(int64_t P, int nw) { return 256 + ((size_t)P * nw * sizeof(Redo) + 256); }

template <int MODE>
static int polish_mode(Table &t, const Cells &c, const double *M, CellPolishArgs a, const uint64_t *vi,
                       const uint64_t *vf, const double *delta, int64_t n, CellWeights w, void *work, cudaStream_t s) {
    using R = PolishRule<MODE>;
    char *q = (char *)work;
    int *d_count = carve<int>(q, 1);
    Redo *list = carve<Redo>(q, (size_t)a.P * a.nw);
    MB_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int), s));
    const dim3 grid((unsigned)a.P, (unsigned)a.nw);
    if (c.n <= CPOL_CELLS) {
        const int bytes = c.n * CPOL_LD * (int)sizeof(double);
        MB_CUDA(cudaFuncSetAttribute(cell_polish_kernel<MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     CPOL_CELLS * CPOL_LD * (int)sizeof(double)));
        cell_polish_kernel<MODE, true><<<grid, cpol_threads(true), bytes, s>>>(c, M, a, delta, list, d_count);
    } else {
        cell_polish_kernel<MODE, false><<<grid, cpol_threads(false), 0, s>>>(c, M, a, delta, list, d_count);
    }
    MB_CUDA(cudaGetLastError());
    int count = 0;
    MB_CUDA(cudaMemcpyAsync(&count, d_count, sizeof(int), cudaMemcpyDeviceToHost, s));
    MB_CUDA(cudaStreamSynchronize(s));
    if (count == 0) return MB_OK;
    t.polish_redone += count;
    RedoBuf rb;
    size_t bn = 0;
    bool room = false;
    for (rb.batch = redo_batch(count, n);; rb.batch /= 2) {
        bn = (size_t)rb.batch * n;
        MB_TRY(t.redo.ensure((2 * rb.batch * sizeof(RedoState) + 256) +
                             (2 * rb.batch * REDO_GROUPS * sizeof(double2) + 256) + 2 * (rb.batch * 8 + 256) +
                             (bn * sizeof(double2) + 256), &room));
        if (room) break;
        if (rb.batch == 1) return NO_ROOM;
    }
    q = (char *)t.redo.p;
    rb.state = carve<RedoState>(q, 2 * (size_t)rb.batch);
    rb.slot = carve<double2>(q, 2 * (size_t)rb.batch * REDO_GROUPS);
    rb.h_best = carve<double>(q, rb.batch);
    rb.d_best = carve<double>(q, rb.batch);
    rb.ab = carve<double2>(q, bn);
    const int ns = MODE == POLISH_SINGLE && a.n_grid == 0 ? 1 : R::starts;
    const ABExact src{view(t), vi, vf, delta};
    for (int e0 = 0; e0 < count; e0 += rb.batch) {
        const unsigned m = (unsigned)std::min(rb.batch, count - e0);
        rb.list = list + e0;
        const unsigned nb = (unsigned)((n + 255) / 256);
        redo_ab_kernel<<<dim3(nb, m), 256, 0, s>>>(src, n, rb);
        for (int st = 0; st < ns; ++st) {
            for (int it = 0; it <= R::iters; ++it)       // the last pass sums h
                redo_pass_kernel<MODE><<<dim3(REDO_GROUPS, m), REDO_THREADS, 0, s>>>(t.d_gamma, n, w, rb, st, it);
            redo_keep_kernel<MODE><<<m, 32, 0, s>>>(rb, a, (int)m, st, st == ns - 1);
        }
        MB_CUDA(cudaGetLastError());
    }
    return MB_OK;
}

int launch_cell_polish(Table &t, const Cells &c, const double *M, const CellPolishArgs &a, const uint64_t *vi,
                       const uint64_t *vf, const double *delta, int64_t n, const CellWeights &w, void *work,
                       cudaStream_t s) {
    if (a.mode == POLISH_EVAL_FAST) return polish_mode<POLISH_EVAL_FAST>(t, c, M, a, vi, vf, delta, n, w, work, s);
    if (a.mode == POLISH_SINGLE) return polish_mode<POLISH_SINGLE>(t, c, M, a, vi, vf, delta, n, w, work, s);
    return polish_mode<POLISH_TOPK>(t, c, M, a, vi, vf, delta, n, w, work, s);
}

}  // namespace mb
