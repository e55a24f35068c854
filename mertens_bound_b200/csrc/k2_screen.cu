// Leaf screen of the lattice enumerators: a staged K2 proxy at 7 offsets.
//
// Reference: ZeroData::fast_screen (search/fast_mertens_enum.cpp:108-142) and the GPU leaf
// scoring of search/gpu_mertens_stream.cu:192-250.  For a leaf y they sum
//   S_m = sum_j 2|c_j| e^{-3e-9 gamma_j^2} cos(gamma_j (y + m 0.0014) + arg c_j),  m = -3..3,
// over the first 64 zeros, reject the leaf if max_m |S_m| is below a threshold, continue over
// zeros 64..127 (and 128..255 on the GPU) with the next threshold, and report the survivors.
// The reference takes cos from a 4096/16384-entry FP32 table at a phase rounded to 12/14 bits
// and the offset as a rounded table step; here the phase is the 32-bit light-tier phase
// (exact to a few units of 2^-32 turn), cos/sin come from MUFU, the offsets are exact
// (frac(step G) from the 128-bit product), and
//   cos(theta + m D) = cos(theta) cos(m D) - sin(theta) sin(m D)
// gives all 7 offsets from one sin/cos pair per (leaf, zero).  Scores agree with the exact sums
// to ~1e-6 of sum |a|; the reference's table proxy is off by up to ~pi/4096 of sum |a|, so the
// two agree on every leaf not within that distance of a threshold.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <type_traits>
#include <vector>

#include "k2_fast.h"
#include "k2_light.cuh"

namespace mb {
namespace {

constexpr int SCREEN_THREADS = 256;
constexpr int SCREEN_MAX_ZEROS = 1024;
constexpr int SCREEN_MAX_STAGES = 8;

// A zero's record: the light phase's limbs (light_phase32_fused where every screened zero has gamma below
// FUSED_PHASE_GAMMA, light_phase32 otherwise) and a cos(2 pi m D), a sin(2 pi m D), m = 1..3, with
// a = 2|c| e^{-k gamma^2} and D = frac(step G).
struct __align__(16) ZScreenF {   // 64 B
    uint32_t b0, b1, psi32;
    float a;
    double b0s, c1s, gh;
    float cm[3], sm[3];
};
struct __align__(16) ZScreenS {   // 80 B
    uint32_t b0, b1, gi, psi32;
    double b0s, c1s, gis, b1s;
    float a, cm[3], sm[3], pad;
};
static_assert(sizeof(ZScreenF) == 64 && sizeof(ZScreenS) == 80, "screen records");

struct ScreenArgs {
    int n_stages;
    int stage_end[SCREEN_MAX_STAGES];
    float thr[SCREEN_MAX_STAGES];
};

struct ScreenOut {
    int64_t max_hits;
    unsigned long long *count;
    int64_t *hit_idx;
    float *hit_score, *scores;
};

MB_DEV void screen_limbs(const TabView &t, int j, ZScreenF &r) {
    const uint32_t b0 = t.g2[j], b1 = t.g3[j];
    r.b0 = b0;
    r.b1 = b1;
    r.psi32 = (uint32_t)((t.psi[j] + 0x80000000ull) >> 32) + 1u;
    r.b0s = u32_to_f64(b0) * TWO_M32;
    r.c1s = u32_to_f64(t.g1[j]) * TWO_M32;
    r.gh = fma(u32_to_f64(t.g4[j]), 4294967296.0, u32_to_f64(b1));
}
MB_DEV void screen_limbs(const TabView &t, int j, ZScreenS &r) {
    const uint32_t b0 = t.g2[j], b1 = t.g3[j], gi = t.g4[j];
    r.b0 = b0;
    r.b1 = b1;
    r.gi = gi;
    r.psi32 = (uint32_t)((t.psi[j] + 0x80000000ull) >> 32) + 2u;
    r.b0s = u32_to_f64(b0) * TWO_M32;
    r.c1s = u32_to_f64(t.g1[j]) * TWO_M32;
    r.gis = u32_to_f64(gi) * TWO_M32;
    r.b1s = u32_to_f64(b1) * TWO_M32;
    r.pad = 0.f;
}
MB_DEV int32_t screen_phase(const CandRegs &c, const ZScreenF &z) {
    return (int32_t)light_phase32_fused(c, z.b0, z.b1, z.b0s, z.c1s, z.gh, z.psi32);
}
MB_DEV int32_t screen_phase(const CandRegs &c, const ZScreenS &z) {
    return (int32_t)light_phase32(c, z.b0, z.b1, z.gi, z.b0s, z.c1s, z.gis, z.b1s, z.psi32);
}

template <class Z>
MB_DEV void screen_sincos(const CandRegs &c, const Z &z, float &sn, float &cs) {
    const float th = (float)screen_phase(c, z) * 1.4629180792671596e-09f;       // 2pi 2^-32
    sn = __sinf(th);
    cs = __cosf(th);
}

// The seven sums of a leaf by parity: S_0 = e[0], S_{+-m} = e[m] -+ o[m - 1]
// (cos(theta + m D) = cos theta cos m D - sin theta sin m D), so a term is seven FMAs.
struct ScreenSums {
    float e[4], o[3];
    MB_DEV void clear() {
        e[0] = e[1] = e[2] = e[3] = o[0] = o[1] = o[2] = 0.f;
    }
    template <class Z>
    MB_DEV void add(const CandRegs &c, const Z &z) {
        float sn, cs;
        screen_sincos(c, z, sn, cs);
        e[0] = fmaf(z.a, cs, e[0]);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            e[m + 1] = fmaf(z.cm[m], cs, e[m + 1]);
            o[m] = fmaf(z.sm[m], sn, o[m]);
        }
    }
    MB_DEV float best() const {
        float b = fabsf(e[0]);
#pragma unroll
        for (int m = 0; m < 3; ++m) b = fmaxf(b, fmaxf(fabsf(e[m + 1] - o[m]), fabsf(e[m + 1] + o[m])));
        return b;
    }
};

// One CTA slot each: an equal share of the leaves, in tiles of LPT x 256.  The first stage runs LPT leaves per thread, so that a
// zero's record (four 16-byte broadcasts) serves LPT terms: with one leaf per thread those reads were half of the
// time (2^20 leaves: 155 us; now 78).  Survivors are listed in shared memory with their sums, and the later
// stages run over the list: a leaf per thread while there are 64 or more (two warps: with a quarter of a
// 1,024-leaf tile as the limit, 200,000 leaves of which a fifth goes on took 105 us, more than one leaf per thread
// throughout, 95; now 40), eight lanes per leaf below that and a warp per leaf from eight leaves down, so a few
// survivors neither hold whole warps nor run a long serial loop: as many zeros' sines and cosines at a time, one
// lane's each, then seven lanes add them in zero order, one sum each.  Every way adds a leaf's terms in the same
// order, so its scores do not depend on the leaves beside it.
template <int LPT, class Z>
__global__ void __launch_bounds__(SCREEN_THREADS, LPT == 1 ? 4 : 2)
screen_kernel(TabView t, int n_zeros, double k, uint64_t step_int, uint64_t step_frac, CandView c, ScreenArgs sa,
              ScreenOut out) {
    constexpr int LEAVES = LPT * SCREEN_THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Z *zs = reinterpret_cast<Z *>(smem_raw);
    float *sums = reinterpret_cast<float *>(smem_raw + (size_t)n_zeros * sizeof(Z));     // [7][LEAVES]
    float *sc = sums + 7 * LEAVES;                                                        // [n_stages][LEAVES]
    uint16_t *list = reinterpret_cast<uint16_t *>(sc + sa.n_stages * LEAVES);             // [2][LEAVES]
    __shared__ int n_list[2];
    __shared__ __align__(16) float trig[SCREEN_THREADS / 32][2][32];     // cosines, sines of a warp's four leaves
    for (int j = threadIdx.x; j < n_zeros; j += SCREEN_THREADS) {
        Z r;
        screen_limbs(t, j, r);
        const double g = t.gamma[j];
        const double a = 2.0 * t.alpha[j] * exp(-k * g * g);
        r.a = (float)a;
        uint64_t hi, lo;
        phase128_exact((uint32_t)step_frac, (uint32_t)(step_frac >> 32), (uint32_t)step_int, (uint32_t)(step_int >> 32),
                       t.g0[j], t.g1[j], t.g2[j], t.g3[j], t.g4[j], hi, lo);
        const double D = s64_turns_to_f64(hi);      // frac(step G) in [-1/2, 1/2)
#pragma unroll
        for (int m = 1; m <= 3; ++m) {
            double s, co;
            sincospi(2.0 * m * D, &s, &co);
            r.cm[m - 1] = (float)(a * co);
            r.sm[m - 1] = (float)(a * s);
        }
        zs[j] = r;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // this CTA's share of the leaves (whole warps of them), tile by tile
    const int64_t warps = (c.P + 31) / 32;
    const int64_t p_end = min(c.P, warps * (blockIdx.x + 1) / gridDim.x * 32);
    for (int64_t p0 = warps * blockIdx.x / gridDim.x * 32; p0 < p_end; p0 += LEAVES) {
        const int n_leaves = (int)min((int64_t)LEAVES, p_end - p0);
        // leaf l's stage result: its score, and the next list or the hit buffers if it survives
        auto finish = [&](int l, int s, const ScreenSums &x) {
            const float b = x.best();
            sc[s * LEAVES + l] = b;
            if (out.scores) out.scores[(p0 + l) * sa.n_stages + s] = b;
            if (!(b >= sa.thr[s])) return;
            if (s + 1 < sa.n_stages) {
                const int q = atomicAdd(&n_list[s & 1], 1);
                list[(s & 1) * LEAVES + q] = (uint16_t)l;
#pragma unroll
                for (int m = 0; m < 4; ++m) sums[m * LEAVES + l] = x.e[m];
#pragma unroll
                for (int m = 0; m < 3; ++m) sums[(4 + m) * LEAVES + l] = x.o[m];
            } else {
                const unsigned long long h = atomicAdd(out.count, 1ull);
                if ((int64_t)h < out.max_hits) {
                    out.hit_idx[h] = p0 + l;
                    for (int i = 0; i < sa.n_stages; ++i) out.hit_score[h * sa.n_stages + i] = sc[i * LEAVES + l];
                }
            }
        };
        auto resume = [&](int l, ScreenSums &x) {
#pragma unroll
            for (int m = 0; m < 4; ++m) x.e[m] = sums[m * LEAVES + l];
#pragma unroll
            for (int m = 0; m < 3; ++m) x.o[m] = sums[(4 + m) * LEAVES + l];
        };
        __syncthreads();                             // the records; the tile before is done with the lists
        if (threadIdx.x < 2) n_list[threadIdx.x] = 0;
        __syncthreads();
        // the first stage with L leaves per thread
        auto first = [&](auto per) {
            constexpr int L = decltype(per)::value;
            CandRegs cr[L];
            ScreenSums x[L];
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const int l = i * SCREEN_THREADS + threadIdx.x;
                cr[i] = cand_regs(c, p0 + l, l < n_leaves);
                x[i].clear();
            }
            for (int j = 0; j < sa.stage_end[0]; ++j) {
                const Z z = zs[j];
#pragma unroll
                for (int i = 0; i < L; ++i) x[i].add(cr[i], z);
            }
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const int l = i * SCREEN_THREADS + threadIdx.x;
                if (l >= n_leaves) continue;
                if (out.scores)
                    for (int s = 1; s < sa.n_stages; ++s) out.scores[(p0 + l) * sa.n_stages + s] = -1.0f;
                finish(l, 0, x[i]);
            }
        };
        if constexpr (LPT == 1) {
            first(std::integral_constant<int, 1>());
        } else {                                     // a last, smaller tile takes fewer per thread
            static_assert(LPT == 4, "one or four leaves per thread");
            if (n_leaves > 3 * SCREEN_THREADS) first(std::integral_constant<int, 4>());
            else if (n_leaves > 2 * SCREEN_THREADS) first(std::integral_constant<int, 3>());
            else if (n_leaves > SCREEN_THREADS) first(std::integral_constant<int, 2>());
            else first(std::integral_constant<int, 1>());
        }
        // the list's n leaves with L lanes each
        auto by_lanes = [&](auto lanes, int n, const uint16_t *in, int s, int j0, int j1) {
            constexpr int L = decltype(lanes)::value, stride = sizeof(Z) / sizeof(float);
            const int g0 = lane & ~(L - 1);              // the leaf's first lane
            const int m = min(lane - g0, 6);             // 0..3: e[m], 4..6: o[m - 4]; lanes above add a copy
            const float *coef = m == 0 ? &zs->a : (m < 4 ? zs->cm + m - 1 : zs->sm + m - 4);
            const float *val = &trig[warp][m < 4 ? 0 : 1][g0];
            for (int q0 = warp * (32 / L); q0 < n; q0 += SCREEN_THREADS / L) {
                const int q = q0 + g0 / L;
                const bool live = q < n;
                const int l = in[live ? q : q0];
                const CandRegs cr = cand_regs(c, p0 + l, true);
                float x = sums[m * LEAVES + l];
                for (int j = j0; j < j1; j += L) {
                    float sn, cs;
                    screen_sincos(cr, zs[min(j + lane - g0, j1 - 1)], sn, cs);
                    __syncwarp();                        // the values before are read
                    trig[warp][0][lane] = cs;
                    trig[warp][1][lane] = sn;
                    __syncwarp();
                    const int nz = min(L, j1 - j);
                    int i = 0;
                    for (; i + 8 <= nz; i += 8) {
                        const float4 u = reinterpret_cast<const float4 *>(val + i)[0];
                        const float4 w = reinterpret_cast<const float4 *>(val + i)[1];
                        const float v[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
                        float a[8];
#pragma unroll
                        for (int b = 0; b < 8; ++b) a[b] = coef[(j + i + b) * stride];
#pragma unroll
                        for (int b = 0; b < 8; ++b) x = fmaf(a[b], v[b], x);
                    }
                    for (; i < nz; ++i) x = fmaf(coef[(j + i) * stride], val[i], x);
                }
                ScreenSums y;
#pragma unroll
                for (int i = 0; i < 4; ++i) y.e[i] = __shfl_sync(0xffffffffu, x, g0 + i);
#pragma unroll
                for (int i = 0; i < 3; ++i) y.o[i] = __shfl_sync(0xffffffffu, x, g0 + 4 + i);
                if (live && lane == g0) finish(l, s, y);
            }
        };
        for (int s = 1; s < sa.n_stages; ++s) {
            __syncthreads();                         // the list of stage s - 1 is complete
            const int n = n_list[(s - 1) & 1];
            if (n == 0) break;
            const uint16_t *in = list + ((s - 1) & 1) * LEAVES;
            const int j0 = sa.stage_end[s - 1], j1 = sa.stage_end[s];
            if (s > 1) {                             // its other half was stage s - 2's
                __syncthreads();
                if (threadIdx.x == 0) n_list[s & 1] = 0;
                __syncthreads();
            }
            if (n >= SCREEN_THREADS / 4) {
                for (int q = threadIdx.x; q < n; q += SCREEN_THREADS) {
                    const int l = in[q];
                    const CandRegs cr = cand_regs(c, p0 + l, true);
                    ScreenSums x;
                    resume(l, x);
                    for (int j = j0; j < j1; ++j) x.add(cr, zs[j]);
                    finish(l, s, x);
                }
            } else if (n > SCREEN_THREADS / 32) {
                by_lanes(std::integral_constant<int, 8>(), n, in, s, j0, j1);
            } else {
                by_lanes(std::integral_constant<int, 32>(), n, in, s, j0, j1);
            }
        }
    }
}

int screen_args(const Table &t, int n_stages, const int64_t *stage_end, const float *threshold, double k,
                int64_t P, int64_t max_hits, const char *who, ScreenArgs &sa) {
    MB_CHECK_ARG(stage_end && threshold, "%s: null stage argument", who);
    MB_CHECK_ARG(P >= 0 && P <= ((int64_t)1 << 31), "%s: P=%lld", who, (long long)P);
    MB_CHECK_ARG(n_stages >= 1 && n_stages <= SCREEN_MAX_STAGES, "%s: n_stages=%d", who, n_stages);
    MB_CHECK_ARG(std::isfinite(k) && k >= 0, "%s: k=%g", who, k);
    MB_CHECK_ARG(max_hits >= 0, "%s: max_hits=%lld", who, (long long)max_hits);
    sa = ScreenArgs{};
    sa.n_stages = n_stages;
    for (int s = 0; s < n_stages; ++s) {
        MB_CHECK_ARG(stage_end[s] >= 1 && stage_end[s] <= SCREEN_MAX_ZEROS && stage_end[s] <= t.n &&
                         (s == 0 || stage_end[s] > stage_end[s - 1]),
                     "%s: stage_end[%d]=%lld must increase within [1, min(%d, n)]", who, s, (long long)stage_end[s],
                     SCREEN_MAX_ZEROS);
        MB_CHECK_ARG(std::isfinite(threshold[s]), "%s: threshold[%d] is not finite", who, s);
        sa.stage_end[s] = (int)stage_end[s];
        sa.thr[s] = threshold[s];
    }
    return MB_OK;
}

template <int LPT, class Z>
int launch_screen_as(const Table &t, CandView c, double k, uint64_t step_int, uint64_t step_frac, const ScreenArgs &sa,
                     const ScreenOut &out, int sms, cudaStream_t st) {
    constexpr int LEAVES = LPT * SCREEN_THREADS;
    const int nz = sa.stage_end[sa.n_stages - 1];
    const auto bytes = [](int zeros, int stages) {
        return (size_t)zeros * sizeof(Z) + (size_t)LEAVES * (7 + stages) * 4 + 2 * LEAVES * sizeof(uint16_t);
    };
    MB_CUDA(cudaFuncSetAttribute(screen_kernel<LPT, Z>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)bytes(SCREEN_MAX_ZEROS, SCREEN_MAX_STAGES)));
    const int64_t tiles = (c.P + LEAVES - 1) / LEAVES;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, (int64_t)sms * (LPT == 1 ? 4 : 2));
    screen_kernel<LPT, Z><<<grid, SCREEN_THREADS, bytes(nz, sa.n_stages), st>>>(view(t), nz, k, step_int, step_frac, c,
                                                                              sa, out);
    MB_CUDA(cudaGetLastError());
    return MB_OK;
}

// The count reset and the screen over P device leaves, on st.  Four leaves per thread where that still gives
// every SM a CTA.
int launch_screen(const Table &t, int64_t P, const uint64_t *d_vi, const uint64_t *d_vf, double k, uint64_t step_int,
                  uint64_t step_frac, const ScreenArgs &sa, const ScreenOut &out, cudaStream_t st) {
    MB_CUDA(cudaMemsetAsync(out.count, 0, 8, st));
    int sms = 148;
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t.device));
    const CandView c{d_vi, d_vf, nullptr, P};
    const bool fused = t.h_gamma[sa.stage_end[sa.n_stages - 1] - 1] < FUSED_PHASE_GAMMA;
    const bool four = P >= (int64_t)sms * 4 * SCREEN_THREADS;
    if (fused)
        return four ? launch_screen_as<4, ZScreenF>(t, c, k, step_int, step_frac, sa, out, sms, st)
                    : launch_screen_as<1, ZScreenF>(t, c, k, step_int, step_frac, sa, out, sms, st);
    return four ? launch_screen_as<4, ZScreenS>(t, c, k, step_int, step_frac, sa, out, sms, st)
                : launch_screen_as<1, ZScreenS>(t, c, k, step_int, step_frac, sa, out, sms, st);
}

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" int mb_screen(mb_table *h, int64_t P, const uint64_t *v_int, const uint64_t *v_frac, double k,
                         uint64_t step_int, uint64_t step_frac, int n_stages, const int64_t *stage_end,
                         const float *threshold, int64_t max_hits, int64_t *out_hits, float *out_hit_scores,
                         int64_t *n_hits, float *out_scores) {
    const char *who = "mb_screen";
    MB_CHECK_ARG(h && v_int && v_frac && stage_end && threshold && n_hits, "%s: null argument", who);
    Table &t = table_of(h);
    MB_CHECK_ARG(max_hits >= 0 && (max_hits == 0 || (out_hits && out_hit_scores)), "%s: hit buffers", who);
    ScreenArgs sa;
    MB_TRY(screen_args(t, n_stages, stage_end, threshold, k, P, max_hits, who, sa));
    *n_hits = 0;
    if (P == 0) return MB_OK;
    MB_TRY(device_guard(t.device));
    const size_t cand = (size_t)P * 8;
    const size_t sc_bytes = out_scores ? (size_t)P * n_stages * 4 : 0;
    const size_t need = 2 * (cand + 256) + 256 + ((size_t)max_hits * 8 + 256) +
                        ((size_t)max_hits * n_stages * 4 + 256) + (sc_bytes + 256);
    MB_TRY(t.io.ensure(need));
    char *q = (char *)t.io.p;
    uint64_t *d_vi = carve<uint64_t>(q, P), *d_vf = carve<uint64_t>(q, P);
    unsigned long long *d_count = carve<unsigned long long>(q, 1);
    int64_t *d_hits = carve<int64_t>(q, max_hits);
    float *d_hsc = carve<float>(q, (size_t)max_hits * n_stages);
    float *d_sc = out_scores ? carve<float>(q, (size_t)P * n_stages) : nullptr;
    cudaStream_t st = t.stream;
    MB_CUDA(cudaMemcpyAsync(d_vi, v_int, cand, cudaMemcpyHostToDevice, st));
    MB_CUDA(cudaMemcpyAsync(d_vf, v_frac, cand, cudaMemcpyHostToDevice, st));
    MB_TRY(launch_screen(t, P, d_vi, d_vf, k, step_int, step_frac, sa, ScreenOut{max_hits, d_count, d_hits, d_hsc, d_sc},
                         st));
    unsigned long long total = 0;
    MB_CUDA(cudaMemcpyAsync(&total, d_count, 8, cudaMemcpyDeviceToHost, st));
    if (out_scores) MB_CUDA(cudaMemcpyAsync(out_scores, d_sc, sc_bytes, cudaMemcpyDeviceToHost, st));
    MB_CUDA(cudaStreamSynchronize(st));
    *n_hits = (int64_t)total;
    const int64_t kept = std::min<int64_t>((int64_t)total, max_hits);
    if (kept > 0) {
        std::vector<int64_t> idx(kept);
        std::vector<float> hs((size_t)kept * n_stages);
        MB_CUDA(cudaMemcpy(idx.data(), d_hits, kept * 8, cudaMemcpyDeviceToHost));
        MB_CUDA(cudaMemcpy(hs.data(), d_hsc, (size_t)kept * n_stages * 4, cudaMemcpyDeviceToHost));
        // the atomic slots come in arbitrary order: return hits sorted by leaf index
        std::vector<int64_t> ord(kept);
        std::iota(ord.begin(), ord.end(), 0);
        std::sort(ord.begin(), ord.end(), [&](int64_t a, int64_t b) { return idx[a] < idx[b]; });
        for (int64_t i = 0; i < kept; ++i) {
            out_hits[i] = idx[ord[i]];
            for (int s = 0; s < n_stages; ++s) out_hit_scores[i * n_stages + s] = hs[ord[i] * n_stages + s];
        }
    }
    if ((int64_t)total > max_hits) {
        set_error("%s: %llu hits exceed max_hits=%lld (the kept subset is arbitrary)", who, total,
                  (long long)max_hits);
        return MB_ERR_CAPACITY;
    }
    return MB_OK;
}

extern "C" int mb_screen_dev(mb_table *h, int64_t P, const uint64_t *d_v_int, const uint64_t *d_v_frac, double k,
                             uint64_t step_int, uint64_t step_frac, int n_stages, const int64_t *stage_end,
                             const float *threshold, int64_t max_hits, int64_t *d_hits, float *d_hit_scores,
                             unsigned long long *d_n_hits, float *d_scores, void *stream) {
    const char *who = "mb_screen_dev";
    MB_CHECK_ARG(h && d_v_int && d_v_frac && d_n_hits, "%s: null argument", who);
    MB_CHECK_ARG(max_hits == 0 || (d_hits && d_hit_scores), "%s: hit buffers", who);
    Table &t = table_of(h);
    ScreenArgs sa;
    MB_TRY(screen_args(t, n_stages, stage_end, threshold, k, P, max_hits, who, sa));
    MB_TRY(device_guard(t.device));
    const cudaStream_t st = (cudaStream_t)stream;
    if (P == 0) {
        MB_CUDA(cudaMemsetAsync(d_n_hits, 0, 8, st));
        return MB_OK;
    }
    return launch_screen(t, P, d_v_int, d_v_frac, k, step_int, step_frac, sa,
                         ScreenOut{max_hits, d_n_hits, d_hits, d_hit_scores, d_scores}, st);
}
