// (cos, sin) of a phase word in turns from a shared-memory table without bank conflicts; used by the plain
// kernel, the heavy tier (its own remainder) and the cell moments.
#pragma once
#include "k2_common.cuh"

namespace mb {

// (cos, sin)(2 pi q / 256) in eight interleaved copies: entry q of copy c sits in the c-th
// 16-byte bank group, and lane l reads copy l mod 8, so a warp's 32 random entries are read in the
// four shared-memory cycles of a conflict-free 512-byte access (one copy of a 2048-entry table: about nine, for
// the random entries' bank conflicts).
constexpr int PH_TAB = 256;
constexpr int PH_COPIES = 8;
constexpr int PH_BYTES = PH_TAB * PH_COPIES * (int)sizeof(double2);

MB_DEV void phasor_table_init(double2 *tab, int threads) {
    for (int i = threadIdx.x; i < PH_TAB; i += threads) {
        double sn, cs;
        sincospi((double)i * (2.0 / PH_TAB), &sn, &cs);
#pragma unroll
        for (int c = 0; c < PH_COPIES; ++c) tab[i * PH_COPIES + c] = make_double2(cs, sn);
    }
}

// cos, sin of the phase word w - 2^51 in units of 2^-60 turn (the top four bits of w are ignored; the caller
// adds 2^51, half a table step): table entry bits [52, 60) of w rotated by d 2^-60 turn,
// d = (w mod 2^52) - 2^51 exact in FP64 (at most 0.0123 rad).  With a = 2 pi 2^-60:
//   sin(a d)     = d (a - a^3 d^2 / 6 + a^5 d^4 / 120)            (truncation 8.4e-18)
//   cos(a d) - 1 = d^2 (-a^2 / 2 + a^4 d^2 / 24 - a^6 d^4 / 720)  (truncation 1.3e-20)
// so the result carries the table's and the last FMA's roundings only.  copy: the lane's copy of the table.
MB_DEV void phasor(uint64_t w, const double2 *copy, double &cs, double &sn) {
    constexpr double a = 6.283185307179586 * 0x1p-60;
    const uint32_t hi = (uint32_t)(w >> 32);
    const double2 T = *reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(copy) +
                                                         ((hi >> 13) & (uint32_t)((PH_TAB - 1) * PH_COPIES * 16)));
    const double d = __hiloint2double((int)((hi & 0xFFFFFu) | 0x43300000u), (int)(uint32_t)w) - 6755399441055744.0;
    const double u = d * d;
    const double s = d * fma(u, fma(u, a * a * a * a * a / 120.0, -a * a * a / 6.0), a);
    const double m = u * fma(u, fma(u, -a * a * a * a * a * a / 720.0, a * a * a * a / 24.0), -a * a / 2.0);
    cs = fma(T.x, m, fma(-T.y, s, T.x));
    sn = fma(T.y, m, fma(T.x, s, T.y));
}

}  // namespace mb
