// Certified interval evaluation of K2 with directed rounding.
//
// Returns [lo, hi] containing the exact value of
//   K2 = 2 sum_{gamma_j < T} exp(-k gamma_j^2) Re(c_j e^{i gamma_j v})
// for the table's exact G_j = gamma_j/2pi (64.128), exact FP64 c_j, gamma_j = 2pi G_j (the FP64
// gamma is within 4 ulp of it, checked at table creation), exact k, and v = v_int + v_frac 2^-64
// widened by an optional radius v_rad.  Term by term (certification/certify_K2.py:116-121
// does the same sum in Arb balls):
//   phase    floor(frac(v G) 2^128), exact; quadrant q from its top two bits; the rest
//            r in [m 2^-62, (m+1) 2^-62] (directed conversions); r > 1/2 uses 1 - r with
//            sine and cosine exchanged, so x = (pi/2) r lies in [0, pi/4 + 2^-60].
//   sin, cos Taylor polynomials of sin x / x (9 terms) and cos x (10 terms) in u = x^2,
//            coefficients as outward-rounded intervals, Horner with __fma_rd / __fma_ru, plus
//            bounds of the Lagrange remainders x^19/19! and x^20/20!.
//   weight   w in [exp(-k gamma_hi^2)(1 - 2^-51), exp(-k gamma_lo^2)(1 + 2^-51)]: CUDA's exp()
//            has a documented maximum error of 1 ulp; the bound allows 2.
//   term     2 w (Re c cos - Im c sin) in interval arithmetic, widened by
//            2 w_hi (|c| gamma_hi v_rad + term_rad_j).
//   sums     per thread, then warp / block / chunk reductions, lower ends with __dadd_rd and
//            upper ends with __dadd_ru.  Also an upper bound of sum 2 w |c| (certify_K2's absS).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "k2_common.cuh"
#include "k2_internal.h"

namespace mb {

struct Ival {
    double lo, hi;
};

// u p + c for u >= 0 and an interval p that is wholly positive (POS) or wholly negative: the lower end of
// u p takes u.lo if p > 0 and u.hi if p < 0, the upper end the other one.  In both series below the partial
// polynomial p_k = c_k + u p_{k+1} has the sign of c_k, (-1)^k: u <= (pi/4)^2 (1 + 2^-58) < 0.617 and
// |c_{k+1} / c_k| <= 1/2, so |u p_{k+1}| <= 0.617 |c_{k+1}| / (1 - 0.31) < 0.45 |c_k|, with the ends'
// roundings far smaller.  (Choosing by comparing the ends costs two FP64 comparisons and four selects a
// step.)
template <bool POS>
MB_DEV Ival horner_step(const Ival &u, const Ival &p, double clo, double chi) {
    return POS ? Ival{__fma_rd(u.lo, p.lo, clo), __fma_ru(u.hi, p.hi, chi)}
               : Ival{__fma_rd(u.hi, p.lo, clo), __fma_ru(u.lo, p.hi, chi)};
}
// p_0 from the leading interval p_K of a series with coefficients (-1)^k |c_k|.
template <int K>
MB_DEV Ival horner(const Ival &u, Ival p, const double *clo, const double *chi) {
    if constexpr (K > 0) return horner<K - 1>(u, horner_step<K % 2 == 0>(u, p, clo[K - 1], chi[K - 1]), clo, chi);
    else return p;
}

// Enclosures of sin x and cos x for x in [x.lo, x.hi], 0 <= x.lo <= x.hi <= pi/4 + 2^-60.
MB_DEV void iv_sincos(const Ival &x, Ival &s, Ival &c) {
    const Ival u{__dmul_rd(x.lo, x.lo), __dmul_ru(x.hi, x.hi)};
    const Ival p = horner<8>(u, Ival{CERT_S_LO[8], CERT_S_HI[8]}, CERT_S_LO, CERT_S_HI);
    // sin x / x >= 0.9 > 0 on this range
    s = {__dmul_rd(x.lo, p.lo), __dmul_ru(x.hi, p.hi)};
    // x^19 / 19! <= x (pi/4 + 2^-60)^18 / 19! < 1.07e-19 x, below half an ulp of sin x
    const double rs = __dmul_ru(x.hi, 1.07e-19);
    s.lo = __dsub_rd(s.lo, rs);
    s.hi = __dadd_ru(s.hi, rs);
    const Ival q = horner<9>(u, Ival{CERT_C_LO[9], CERT_C_HI[9]}, CERT_C_LO, CERT_C_HI);
    const double rc = 3.3e-21;                     // >= (pi/4 + 2^-60)^20 / 20!
    c = {__dsub_rd(q.lo, rc), __dadd_ru(q.hi, rc)};
}

// point * interval
MB_DEV Ival iv_scale(double a, const Ival &b) {
    const bool neg = __double2hiint(a) < 0;
    return {__dmul_rd(a, neg ? b.hi : b.lo), __dmul_ru(a, neg ? b.lo : b.hi)};
}

// non-negative interval w times interval a
MB_DEV Ival iv_wmul(const Ival &w, const Ival &a) {
    double lo = a.lo >= 0.0 ? __dmul_rd(w.lo, a.lo) : __dmul_rd(w.hi, a.lo);
    double hi = a.hi >= 0.0 ? __dmul_ru(w.hi, a.hi) : __dmul_ru(w.lo, a.hi);
    return {lo, hi};
}

// Enclosure of exp(-y) for y in [ylo, yhi], 0 <= ylo <= yhi.
MB_DEV Ival iv_exp_neg(double ylo, double yhi) {
    const double e_big = exp(-ylo);
    // a narrow y: exp(-yhi) >= exp(-ylo) (1 - d), below it by at most d^2 / 2 < 2^-57 relative, and
    // (1 - 2^-51)(1 - d) >= 1 - (2^-51 + d): one exponential for both ends
    const double d = __dsub_ru(yhi, ylo);
    if (d < 0x1p-28 && e_big > 1e-300)
        return {__fma_rd(-e_big, __dadd_ru(d, 0x1p-51), e_big), __dmul_ru(e_big, 1.0 + 0x1p-51)};
    const double e_small = exp(-yhi);
    const double tiny = 4.0 * 4.9406564584124654e-324;     // absolute slack in the subnormal range
    double lo = __dmul_rd(e_small, 1.0 - 4.440892098500626e-16);
    double hi = __dmul_ru(e_big, 1.0 + 4.440892098500626e-16);
    if (e_small < 2.2250738585072014e-308) lo = fmax(0.0, __dsub_rd(lo, tiny));
    if (e_big < 2.2250738585072014e-308) hi = __dadd_ru(hi, tiny);
    return {lo, hi};
}

// One zero's data; rad: its term's own radius.
struct CertZero {
    uint32_t g0, g1, g2, g3, g4;
    double gamma, cr, ci, rad;
};

MB_DEV CertZero cert_zero(const TabView &tv, int64_t j, const double *term_rad, int64_t jr) {
    return {tv.g0[j], tv.g1[j], tv.g2[j], tv.g3[j], tv.g4[j], tv.gamma[j], tv.cre[j], tv.cim[j],
            term_rad ? term_rad[jr] : 0.0};
}

// What a zero's terms share over the candidates: gamma and the weight enclosed, |c| rounded up.
struct CertWeight {
    double glo, ghi, cabs;
    Ival w;
};

// k lies in [k_lo, k_hi].
MB_DEV CertWeight cert_weight(const CertZero &z, double k_lo, double k_hi) {
    CertWeight x;
    x.glo = __dmul_rd(z.gamma, 1.0 - 8.881784197001252e-16);
    x.ghi = __dmul_ru(z.gamma, 1.0 + 8.881784197001252e-16);
    x.w = iv_exp_neg(__dmul_rd(__dmul_rd(k_lo, x.glo), x.glo), __dmul_ru(__dmul_ru(k_hi, x.ghi), x.ghi));
    x.cabs = __dsqrt_ru(__fma_ru(z.cr, z.cr, __dmul_ru(z.ci, z.ci)));
    return x;
}

struct CertTerm {
    Ival t;         // 2 w Re(c e^{i theta})
    double abs_hi;  // 2 w |c| rounded up
    Ival dd, dk;    // -2 w gamma Im(c e^{i theta}) and -2 w gamma^2 Re(c e^{i theta}) (GRAD only)
};

// -2 x for an interval x (exact)
MB_DEV Ival iv_m2(const Ival &x) { return {-2.0 * x.hi, -2.0 * x.lo}; }

// One zero's term for one candidate.  With GRAD its derivatives in v (= delta) and k are enclosed too:
//   d/dv 2 w Re(c e^{i gamma v}) = -2 w gamma Im(c e^{i gamma v}) = -2 w gamma (Re c sin + Im c cos),
//   d/dk 2 w Re(c e^{i gamma v}) = -2 w gamma^2 Re(c e^{i gamma v}),
// from the same sine/cosine and weight intervals and gamma in [gamma_lo, gamma_hi]; a radius rho
// of c e^{i gamma v} (|c| gamma_hi v_rad + term_rad) widens them by 2 w_hi gamma_hi rho and
// 2 w_hi gamma_hi^2 rho (each derivative in v brings one more factor gamma).
// weight() gives the zero's CertWeight; it is called behind the sines, whose registers it can then take.
template <bool GRAD, class Weight>
MB_DEV CertTerm cert_term(const CertZero &z, Weight weight, uint64_t vi, uint64_t vf, double v_rad) {
    uint64_t hi, lo;
    phase128_exact((uint32_t)vf, (uint32_t)(vf >> 32), (uint32_t)vi, (uint32_t)(vi >> 32), z.g0, z.g1, z.g2, z.g3,
                   z.g4, hi, lo);
    const int q = (int)(hi >> 62);
    const uint64_t m = hi & ((1ull << 62) - 1);
    const double two_m62 = 2.168404344971009e-19;
    Ival r{__ull2double_rd(m) * two_m62, __ull2double_ru(m + 1) * two_m62};
    bool swap = false;
    if (r.lo >= 0.5) {
        r = {__dsub_rd(1.0, r.hi), __dsub_ru(1.0, r.lo)};
        swap = true;
    }
    Ival s, c;
    iv_sincos(Ival{__dmul_rd(CERT_PIO2_LO, r.lo), __dmul_ru(CERT_PIO2_HI, r.hi)}, s, c);
    // c e^{i theta} over the octant's s and c: the quadrant's signs (q = 0: cos, sin = c, s; 1: -s, c;
    // 2: -c, -s; 3: s, -c) and its exchange go into the point coefficients
    const double cr = z.cr, ci = z.ci;
    const bool nc = q == 1 || q == 2, ns = q >= 2;                 // cos and sin negated
    const bool ex = swap != ((q & 1) != 0);
    const double rc = nc ? -cr : cr, rs = ns ? ci : -ci;           // Re = rc cos' + rs sin'
    const Ival a1 = iv_scale(ex ? rc : rs, s), a2 = iv_scale(ex ? rs : rc, c);
    const Ival A{__dadd_rd(a1.lo, a2.lo), __dadd_ru(a1.hi, a2.hi)};
    const CertWeight x = weight();
    const Ival &w = x.w;
    const double glo = x.glo, ghi = x.ghi, cabs = x.cabs;
    Ival t = iv_wmul(w, A);
    t.lo *= 2.0;
    t.hi *= 2.0;
    double rad = 0.0;
    if (v_rad > 0.0) rad = __dmul_ru(__dmul_ru(cabs, ghi), v_rad);
    if (z.rad != 0.0) rad = __dadd_ru(rad, z.rad);
    double wr = 0.0;
    if (rad > 0.0) {
        wr = __dmul_ru(2.0 * w.hi, rad);
        t.lo = __dsub_rd(t.lo, wr);
        t.hi = __dadd_ru(t.hi, wr);
    }
    CertTerm out{t, __dmul_ru(2.0 * w.hi, cabs), {0.0, 0.0}, {0.0, 0.0}};
    if constexpr (GRAD) {
        const double ic = nc ? -ci : ci, is = ns ? -cr : cr;       // Im = ic cos' + is sin'
        const Ival b1 = iv_scale(ex ? ic : is, s), b2 = iv_scale(ex ? is : ic, c);
        const Ival B{__dadd_rd(b1.lo, b2.lo), __dadd_ru(b1.hi, b2.hi)};
        const Ival wg{__dmul_rd(w.lo, glo), __dmul_ru(w.hi, ghi)};          // w gamma >= 0
        const Ival wg2{__dmul_rd(wg.lo, glo), __dmul_ru(wg.hi, ghi)};      // w gamma^2 >= 0
        out.dd = iv_m2(iv_wmul(wg, B));
        out.dk = iv_m2(iv_wmul(wg2, A));
        if (wr > 0.0) {
            const double r1 = __dmul_ru(wr, ghi), r2 = __dmul_ru(r1, ghi);
            out.dd = {__dsub_rd(out.dd.lo, r1), __dadd_ru(out.dd.hi, r1)};
            out.dk = {__dsub_rd(out.dk.lo, r2), __dadd_ru(out.dk.hi, r2)};
        }
    }
    return out;
}

constexpr int CERT_THREADS = 256;

// Number of sums per (block, candidate): lo/hi of K2 and abs_hi, plus lo/hi of both derivatives.
template <bool GRAD>
__host__ __device__ constexpr int cert_sums() { return GRAD ? 7 : 3; }

// Upper ends and abs_hi round up, lower ends down.
__host__ __device__ constexpr bool cert_up(int q) { return q == 1 || q == 2 || q == 4 || q == 6; }

// The CTA's directed-rounding sums, in thread 0's acc: the warps' shuffle trees, then the warps in order.
template <int NS>
MB_DEV void cert_block_sum(double (&acc)[NS], double (*red)[NS]) {
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const double x = __shfl_xor_sync(0xffffffffu, acc[q], o);
            acc[q] = cert_up(q) ? __dadd_ru(acc[q], x) : __dadd_rd(acc[q], x);
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NS; ++q) red[warp][q] = acc[q];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            double v = 0.0;
            for (int w = 0; w < CERT_THREADS / 32; ++w) v = cert_up(q) ? __dadd_ru(v, red[w][q]) : __dadd_rd(v, red[w][q]);
            acc[q] = v;
        }
}

// Bound: instruction issue and, with one candidate, the latency of its nine loads per zero: a zero's data are
// loaded one zero ahead, which takes the registers of a fourth CTA per SM and is still the better side (kernel
// 49 -> 44 us for one candidate over 2.3 M zeros).  C candidates share a zero's loads, weight and |c|.
// grid (zero blocks, candidate tiles); partial[(blockIdx.x * P + p) * NS + s] with s = K2 lo, K2 hi,
// abs_hi[, dd lo, dd hi, dk lo, dk hi]: lower ends summed with __dadd_rd, upper ends with __dadd_ru.
template <bool GRAD, int C>
__global__ void __launch_bounds__(CERT_THREADS, C == 1 ? 3 : 2)
k2_certified_kernel(TabView tv, const uint64_t *vi, const uint64_t *vf, const double *v_rad, int64_t P, int64_t j0,
                    int64_t j1, double k_lo, double k_hi, const double *term_rad, double *partial) {
    constexpr int NS = cert_sums<GRAD>();
    const int64_t p0 = (int64_t)blockIdx.y * C;
    const int live = (int)min((int64_t)C, P - p0);
    uint64_t a[C], b[C];
    double acc[C][NS];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int64_t p = p0 + min(i, live - 1);
        a[i] = vi[p];
        b[i] = vf[p];
#pragma unroll
        for (int q = 0; q < NS; ++q) acc[i][q] = 0.0;
    }
    const int64_t stride = (int64_t)gridDim.x * CERT_THREADS;
    int64_t jr = (int64_t)blockIdx.x * CERT_THREADS + threadIdx.x;
    CertZero nxt;
    if (j0 + jr < j1) nxt = cert_zero(tv, j0 + jr, term_rad, jr);
    while (j0 + jr < j1) {
        const CertZero z = nxt;
        jr += stride;
        if (j0 + jr < j1) nxt = cert_zero(tv, j0 + jr, term_rad, jr);
        CertWeight x;
        if constexpr (C > 1) x = cert_weight(z, k_lo, k_hi);
        const auto weight = [&] {
            if constexpr (C > 1) return x;
            else return cert_weight(z, k_lo, k_hi);
        };
#pragma unroll
        for (int i = 0; i < C; ++i) {
            if (i >= live) break;
            const CertTerm ct = cert_term<GRAD>(z, weight, a[i], b[i], v_rad ? v_rad[p0 + i] : 0.0);
            acc[i][0] = __dadd_rd(acc[i][0], ct.t.lo);
            acc[i][1] = __dadd_ru(acc[i][1], ct.t.hi);
            acc[i][2] = __dadd_ru(acc[i][2], ct.abs_hi);
            if constexpr (GRAD) {
                acc[i][3] = __dadd_rd(acc[i][3], ct.dd.lo);
                acc[i][4] = __dadd_ru(acc[i][4], ct.dd.hi);
                acc[i][5] = __dadd_rd(acc[i][5], ct.dk.lo);
                acc[i][6] = __dadd_ru(acc[i][6], ct.dk.hi);
            }
        }
    }
    __shared__ double red[CERT_THREADS / 32][NS];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        if (i >= live) break;
        if (i > 0) __syncthreads();                  // thread 0 has read the sums before
        cert_block_sum<NS>(acc[i], red);
        if (threadIdx.x == 0) {
            double *o = partial + ((int64_t)blockIdx.x * P + p0 + i) * NS;
#pragma unroll
            for (int q = 0; q < NS; ++q) o[q] = acc[i][q];
        }
    }
}

// out[s * P + p] for the NS sums of candidate p (the same order as the partials).  One CTA per candidate:
// a strided directed-rounding sum per thread, then the warps' shuffle trees and the warps in order.  (One
// thread per candidate spent 118 of the 176 us of the 2.3 M-zero, one-candidate interval here: 3,552
// dependent loads.  Now 5 us.)
template <bool GRAD>
__global__ void __launch_bounds__(CERT_THREADS)
certified_reduce_kernel(const double *partial, int64_t P, int nblk, double *out) {
    constexpr int NS = cert_sums<GRAD>();
    __shared__ double red[CERT_THREADS / 32][NS];
    const int64_t p = blockIdx.x;
    double acc[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) acc[q] = 0.0;
    for (int b = threadIdx.x; b < nblk; b += CERT_THREADS)
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const double x = partial[((int64_t)b * P + p) * NS + q];
            acc[q] = cert_up(q) ? __dadd_ru(acc[q], x) : __dadd_rd(acc[q], x);
        }
    cert_block_sum<NS>(acc, red);
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NS; ++q) out[q * P + p] = acc[q];
}

// out (device, NS x P): rows K2 lo, K2 hi, abs_hi [, dd lo, dd hi, dk lo, dk hi].
int launch_certified(Table &t, const uint64_t *d_vi, const uint64_t *d_vf, const double *d_vrad, int64_t P,
                     int64_t j0, int64_t j1, double k_lo, double k_hi, const double *d_term_rad, bool grad,
                     double *d_out, cudaStream_t s) {
    if (P == 0) return MB_OK;
    const int64_t n_use = std::max<int64_t>(0, j1 - j0);
    int sms = 148;
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t.device));
    // four candidates per thread share a third of the work (24 x 400,000: 185 -> 138 us, 4 x 1,000,000: 101 -> 88).
    // 12 CTAs per SM (four rounds of three): longer chains of directed sums would widen the intervals.
    const int C = P >= 4 ? 4 : 1;
    const int64_t n_tile = (P + C - 1) / C;
    const int64_t want = std::max<int64_t>(1, ((int64_t)sms * 12 + n_tile - 1) / n_tile);
    const int64_t nblk = std::max<int64_t>(1, std::min(want, (n_use + CERT_THREADS - 1) / CERT_THREADS));
    MB_CHECK_ARG(P <= 65535, "certified: P=%lld exceeds 65535 candidates per call", (long long)P);
    const int ns = grad ? cert_sums<true>() : cert_sums<false>();
    MB_TRY(t.work.ensure((size_t)nblk * P * ns * sizeof(double)));
    double *partial = (double *)t.work.p;
    const dim3 grid((unsigned)nblk, (unsigned)n_tile);
    auto launch = [&](auto kernel, auto reduce) -> int {
        kernel<<<grid, CERT_THREADS, 0, s>>>(view(t), d_vi, d_vf, d_vrad, P, j0, j1, k_lo, k_hi, d_term_rad, partial);
        MB_CUDA(cudaGetLastError());
        reduce<<<(unsigned)P, CERT_THREADS, 0, s>>>(partial, P, (int)nblk, d_out);
        MB_CUDA(cudaGetLastError());
        return MB_OK;
    };
    if (grad)
        return C == 1 ? launch(k2_certified_kernel<true, 1>, certified_reduce_kernel<true>)
                      : launch(k2_certified_kernel<true, 4>, certified_reduce_kernel<true>);
    return C == 1 ? launch(k2_certified_kernel<false, 1>, certified_reduce_kernel<false>)
                  : launch(k2_certified_kernel<false, 4>, certified_reduce_kernel<false>);
}

}  // namespace mb

using namespace mb;

namespace {

// The shared body of the certified entry points: checks, staging, launch, copy-out of
// out_rows[r] (host, P each) from the NS device rows (null entries are skipped).
int certified_call(const char *who, mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                   const double *v_rad, double k_lo, double k_hi, int64_t j0, int64_t j1, const double *term_rad,
                   bool grad, double *const *out_rows) {
    MB_CHECK_ARG(h && v_int && v_frac, "%s: null argument", who);
    MB_CHECK_ARG(P >= 0 && P <= 65535, "%s: P=%lld out of range (0..65535)", who, (long long)P);
    MB_CHECK_ARG(std::isfinite(k_lo) && std::isfinite(k_hi) && 0.0 <= k_lo && k_lo <= k_hi,
                 "%s: k interval [%g, %g]", who, k_lo, k_hi);
    if (P == 0) return MB_OK;
    Table &t = table_of(h);
    MB_CHECK_ARG(0 <= j0 && j0 <= j1 && j1 <= t.n, "%s: zero range [%lld, %lld) of %lld", who, (long long)j0,
                 (long long)j1, (long long)t.n);
    const int64_t n_use = j1 - j0;
    if (v_rad)
        for (int64_t p = 0; p < P; ++p)
            MB_CHECK_ARG(std::isfinite(v_rad[p]) && v_rad[p] >= 0.0, "%s: v_rad[%lld]", who, (long long)p);
    if (term_rad)
        for (int64_t j = 0; j < n_use; ++j)
            MB_CHECK_ARG(std::isfinite(term_rad[j]) && term_rad[j] >= 0.0, "%s: term_rad[%lld]", who, (long long)j);
    MB_TRY(device_guard(t.device));
    const int ns = grad ? cert_sums<true>() : cert_sums<false>();
    const size_t cb = (size_t)P * 8, rb = term_rad ? (size_t)n_use * 8 : 0;
    MB_TRY(t.io.ensure((3 + ns) * cb + rb + 256));
    char *base = (char *)t.io.p;
    uint64_t *d_vi = (uint64_t *)base, *d_vf = (uint64_t *)(base + cb);
    double *d_vrad = (double *)(base + 2 * cb), *d_out = (double *)(base + 3 * cb);
    double *d_rad = term_rad ? (double *)(base + (3 + ns) * cb) : nullptr;
    // one copy for the candidates, one for all result rows (each small pageable copy costs microseconds)
    std::vector<char> in((v_rad ? 3 : 2) * cb);
    std::memcpy(in.data(), v_int, cb);
    std::memcpy(in.data() + cb, v_frac, cb);
    if (v_rad) std::memcpy(in.data() + 2 * cb, v_rad, cb);
    MB_CUDA(cudaMemcpyAsync(d_vi, in.data(), in.size(), cudaMemcpyHostToDevice, t.stream));
    if (term_rad && rb) MB_CUDA(cudaMemcpyAsync(d_rad, term_rad, rb, cudaMemcpyHostToDevice, t.stream));
    MB_TRY(launch_certified(t, d_vi, d_vf, v_rad ? d_vrad : nullptr, P, j0, j1, k_lo, k_hi, d_rad, grad, d_out,
                            t.stream));
    std::vector<double> rows((size_t)ns * P);
    MB_CUDA(cudaMemcpyAsync(rows.data(), d_out, ns * cb, cudaMemcpyDeviceToHost, t.stream));
    MB_CUDA(cudaStreamSynchronize(t.stream));
    for (int r = 0; r < ns; ++r)
        if (out_rows[r]) std::memcpy(out_rows[r], rows.data() + (size_t)r * P, cb);
    return MB_OK;
}

}  // namespace

extern "C" int mb_k2_certified_range(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                     const double *v_rad, double k_lo, double k_hi, int64_t j0, int64_t j1,
                                     const double *term_rad, double *out_lo, double *out_hi, double *out_abs_hi) {
    MB_CHECK_ARG(out_lo && out_hi, "mb_k2_certified_range: null argument");
    double *rows[3] = {out_lo, out_hi, out_abs_hi};
    return certified_call("mb_k2_certified_range", h, P, v_int, v_frac, v_rad, k_lo, k_hi, j0, j1, term_rad, false,
                          rows);
}

extern "C" int mb_k2_certified_grad_range(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                                          const double *v_rad, double k_lo, double k_hi, int64_t j0, int64_t j1,
                                          const double *term_rad, double *out_lo, double *out_hi) {
    MB_CHECK_ARG(out_lo && out_hi, "mb_k2_certified_grad_range: null argument");
    double *rows[7] = {out_lo, out_hi, nullptr, out_lo + P, out_hi + P, out_lo + 2 * P, out_hi + 2 * P};
    return certified_call("mb_k2_certified_grad_range", h, P, v_int, v_frac, v_rad, k_lo, k_hi, j0, j1, term_rad,
                          true, rows);
}

extern "C" int mb_k2_certified(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac,
                               const double *v_rad, double k, double T, const double *term_rad,
                               double *out_lo, double *out_hi, double *out_abs_hi) {
    MB_CHECK_ARG(h, "mb_k2_certified: null table");
    MB_CHECK_ARG(std::isfinite(k) && k >= 0.0, "mb_k2_certified: k=%g", k);
    MB_CHECK_ARG(!std::isnan(T), "mb_k2_certified: T is NaN");
    return mb_k2_certified_range(h, P, v_int, v_frac, v_rad, k, k, 0, table_of(h).count_below(T), term_rad, out_lo,
                                 out_hi, out_abs_hi);
}
