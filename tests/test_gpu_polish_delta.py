"""The part of a candidate's delta below 2^-64 in the polishes on cell moments.  The moments are taken at v + delta rounded
to 2^-64; gamma times what the rounding dropped, up to 1.4e-13 rad here, has to come back in every value.

Weights of 1e-26 keep |h''| below the 1e-12 at which Newton stops, so h_pol is h at the starting offset 0 (and the only
grid point of the Taylor polish is 0): h_unpol and h_pol are both sum w A.  Per unit of sum 2|c| w the moment terms
carry 4e-16 (phasor) + 5.1e-16 (series) + 3e-16 (sums), A itself 6e-16: below 2e-15."""
import math

import numpy as np
import pytest

from mertens_bound_b200 import k2, path1, synth

pytestmark = pytest.mark.gpu


def _deltas(kind, P, rng):
    sign = rng.choice([-1.0, 1.0], P)
    if kind == "tie":                                           # odd multiples of 2^-65: the rounding is a tie
        return sign * (2.0 * rng.integers(2**51, 2**52, P) + 1.0) * 2.0**-65
    return sign * rng.uniform(1e-6, 1e-5, P)                    # last bits at 2^-72: any rest


@pytest.mark.parametrize("kind", ["rest", "tie"])
def test_rest_of_delta(gpu, small_table, kind):
    rng = np.random.default_rng(91)
    gam = 5.0e6 + np.cumsum(rng.uniform(0.2, 0.72, 3000))
    G3 = synth.fixed_from_double(gam / (2.0 * math.pi), rng)
    data = synth.ZeroTableData(G3, synth.gamma_from_fixed(G3), small_table.c_re[:3000].copy(),
                               small_table.c_im[:3000].copy(), small_table.seed)
    c = synth.make_candidates(40, seed=92)
    c.delta[:] = _deltas(kind, c.n, rng)
    w = np.full(data.n, 1e-26)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(w)
        A, _ = path1.compute_exact_AB(t, c)
        want = np.array([math.fsum(a * w) for a in A])
        tol = 2e-15 * math.fsum(2.0 * np.hypot(data.c_re, data.c_im) * w)
        for got in (path1.polish_peaks_exact(t, c, s, None, 2.5e-4, 0), path1.polish_single_exact(t, c, s, None, 4e-5, 0),
                    path1.fast_polish_exact(t, c, s, None, ddy_grid=np.zeros(1), top=0),
                    path1.fast_polish_exact(t, c, s, None, ddy_grid=np.zeros(1), top=c.n)):
            assert np.max(np.abs(got[0] - want)) <= tol
            assert np.max(np.abs(got[1] - want)) <= tol


@pytest.mark.parametrize("end", ["low", "high"])
def test_sum_outside_the_fixed_point_range(gpu, small_table, end):
    """v + delta below 0 or at 2^64 and above: as on the exact (A, B) of that sum, and for the peaks beside it too."""
    from mertens_bound_b200 import compat
    data = small_table.truncate(3000)
    c = synth.make_candidates(20, seed=93)
    c.delta[:] = np.random.default_rng(93).uniform(-1e-4, 1e-4, c.n)
    c.v_int[:3] = 0 if end == "low" else 2**64 - 1
    c.v_frac[:3] = np.array([12345, 2**40, 2**62] if end == "low" else [2**64 - 2, 2**64 - 2**40, 2**63], np.uint64)
    c.delta[:3] = np.array([-1e-4, -0.7, -60000.0]) * (1 if end == "low" else -1)
    w = np.exp(-3e-9 * data.gamma**2)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(w)
        A, B = path1.compute_exact_AB(t, c)
        one, many = path1.polish_peaks_exact(t, c, s), path1.polish_peaks_weights(t, c, [s, s])
        single, fast = path1.polish_single_exact(t, c, s), path1.fast_polish_exact(t, c, s, top=c.n)
    peaks = compat.polish_peaks_with_weights(A, B, data.gamma, w, 2.5e-4, 40)
    for got, want in ((one, peaks), ([x[1] for x in many], peaks),
                      (single, path1.polish_single_peak(A, B, data.gamma, w)),
                      (fast, path1.fast_polish_batch(A, B, data.gamma, w, top=c.n))):
        for g, x, tol in zip(got, want, (3e-13, 3e-11, 1e-12)):
            np.testing.assert_allclose(g, x, rtol=0, atol=tol)
