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


def test_newton_offsets(gpu, oracle):
    """The Newton offsets of the top peaks against the same four steps in extended precision on the oracle's (A, B): their rms
    error is at most 1.5 times the matrix form's (each rms over some 60 peaks is itself good to a tenth)."""
    n, P = 50_000, 96
    data = synth.make_table(600_000).truncate(n)
    c = synth.make_candidates(P, seed=6)
    w = score.reference_weights(data.gamma)["jp"]
    A, B = oracle.exact_AB(c, data, n)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(w)
        start = path1.fast_polish_exact(t, c, s, top=0)[2]
        got = path1.fast_polish_exact(t, c, s, top=P)[2]
    ref = path1.fast_polish_batch(A, B, data.gamma, w, top=P)[2]
    L = np.longdouble
    g, wl = data.gamma.astype(L), w.astype(L)
    e, f = [], []
    for i in np.flatnonzero((got != 0.0) & (ref != 0.0)):
        x, a, b = L(start[i]), A[i].astype(L), B[i].astype(L)
        for _ in range(4):
            cs, sn = np.cos(g * x), np.sin(g * x)
            step = (wl * g * (-a * sn - b * cs)).sum() / -(wl * g * g * (a * cs - b * sn)).sum()
            step = min(max(step, L(-1e-5)), L(1e-5))
            x -= step
            if abs(step) < 1e-13:
                break
        e.append(float(got[i] - x))
        f.append(float(ref[i] - x))
    assert len(e) > 30
    assert np.sqrt(np.mean(np.square(e))) <= 1.5 * np.sqrt(np.mean(np.square(f)))
