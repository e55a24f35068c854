"""The Taylor polish's grid stage against sums of the oracle's (A, B) in extended precision: its error is not above that of
the matrix form, which adds the same oracle's (A, B) by 2,048 running sums."""
from math import factorial

import numpy as np
import pytest

from mertens_bound_b200 import k2, path1, score, synth

pytestmark = pytest.mark.gpu


def test_error_not_above_the_matrix_form(gpu, oracle):
    n, P = 100_000, 96
    data = synth.make_table(600_000).truncate(n)
    c = synth.make_candidates(P, seed=5)
    w = score.reference_weights(data.gamma)["jp"]
    A, B = oracle.exact_AB(c, data, n)
    L = np.longdouble
    u, wl, z = data.gamma.astype(L) * L(1e-4), w.astype(L), path1.default_grid().astype(L) * L(1e4)
    h = 0
    for m in range(9):
        x = (A.astype(L) * (wl * u**(2 * m))).sum(1) * (-1)**m / L(factorial(2 * m))
        if m == 0:
            h0 = x
        h = h + x[:, None] * z**(2 * m)
        if m < 8:
            y = (B.astype(L) * (wl * u**(2 * m + 1))).sum(1) * (-1)**m / L(factorial(2 * m + 1))
            h = h - y[:, None] * z**(2 * m + 1)
    with k2.ZeroTable.from_data(data) as t:
        got = path1.fast_polish_exact(t, c, t.add_weights(w), top=0)
    ref = path1.fast_polish_batch(A, B, data.gamma, w, top=0)
    j = [int(np.flatnonzero(path1.default_grid() == d)[0]) for d in got[2]]
    assert np.array_equal(got[2], ref[2])
    rms = lambda e: float(np.sqrt(np.mean(np.square(e.astype(float)))))  # noqa: E731
    assert rms(got[0] - h0) <= rms(ref[0] - h0)
    assert rms(got[1] - h[np.arange(P), j]) <= rms(ref[1] - h[np.arange(P), j])
