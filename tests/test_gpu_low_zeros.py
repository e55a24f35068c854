"""Polishes on cell moments over few zeros far below the width that a cell could have: gamma between 1e-3 and 1e-2, where a cell
for the polishes' offsets would be 1e4 times as wide.  Newton's sums are then formed about a centre at the zeros."""
from fractions import Fraction

import numpy as np
import pytest

from mertens_bound_b200 import compat, k2, path1, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 14])
def test_tiny_gamma(gpu, n):
    rng = np.random.default_rng(n)
    gam = 1e-3 + np.cumsum(rng.uniform(1e-5, 1e-3, n))
    G3 = np.empty((n, 3), np.uint64)
    for j, x in enumerate(gam / (2 * np.pi)):
        q = int(Fraction(float(x)) * 2**128)
        G3[j] = (q >> 128, (q >> 64) & (2**64 - 1), q & (2**64 - 1))
    g = synth.gamma_from_fixed(G3)
    data = synth.ZeroTableData(G3, g, rng.standard_normal(n), rng.standard_normal(n), 0)
    c = synth.make_candidates(60, seed=n)
    w = rng.uniform(0.5, 1.0, n)
    grid = np.linspace(-2.5e-4, 2.5e-4, 41)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(w)
        A, B = path1.compute_exact_AB(t, c)
        got = (path1.polish_peaks_exact(t, c, s), path1.polish_single_exact(t, c, s),
               path1.fast_polish_exact(t, c, s, ddy_grid=grid, top=c.n))
    want = (compat.polish_peaks_with_weights(A, B, g, w, 2.5e-4, 40), path1.polish_single_peak(A, B, g, w),
            path1.fast_polish_batch(A, B, g, w, ddy_grid=grid, top=c.n))
    for x, y in zip(got, want):
        for a, b, tol in zip(x, y, (1e-14, 1e-14, 1e-12)):
            np.testing.assert_allclose(a, b, rtol=0, atol=tol * max(1.0, 2 * np.hypot(data.c_re, data.c_im).sum()))
