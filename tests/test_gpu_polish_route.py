"""Polishes on cell moments or over the zeros: the cells' number decides, by each loop's measured break-even."""
import ctypes as C

import numpy as np
import pytest

from mertens_bound_b200 import compat, k2, path1, synth
from mertens_bound_b200._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def full(gpu):
    return synth.make_table(600_000, seed=1)


def _on_cells(table):
    n = C.c_int64()
    check(lib().mb_table_polish_redone(table.handle, C.byref(n)))
    return n.value >= 0


# zeros, half width, and whether peaks / single / top go over the cells
@pytest.mark.parametrize("n,half,want", [
    (600_000, 2.5e-4, (True, True, True)), (600_000, 0.018, (True, True, True)), (600_000, 0.03, (False, True, True)),
    (600_000, 0.08, (False, False, False)), (100_000, 0.01, (True, True, True)), (100_000, 0.03, (True, True, False)),
    (100_000, 0.08, (False, False, False)), (20_000, 0.05, (True, False, False)), (20_000, 0.08, (False, False, False)),
    (3000, 0.08, (True, True, True)), (300, 0.08, (False, False, False)), (60, 0.08, (True, True, True)),
])
def test_route(full, n, half, want):
    data = full.truncate(n)
    c = synth.make_candidates(2, seed=95)
    w = np.exp(-3e-9 * data.gamma**2)
    with k2.ZeroTable.from_data(data) as t:
        s, s2 = t.add_weights(w), t.add_weights(0.5 * w)
        got = path1.polish_peaks_exact(t, c, s, n, half, 2)
        route = [_on_cells(t)]
        both = path1.polish_peaks_weights(t, c, [s, s2], n, half, 2)
        assert _on_cells(t) == route[0]                    # whatever the number of vectors
        one = path1.polish_single_exact(t, c, s, n, half, 2)
        route.append(_on_cells(t))
        path1.fast_polish_exact(t, c, s, n, np.linspace(-half, half, 3), top=2)
        route.append(_on_cells(t))
        A, B = path1.compute_exact_AB(t, c, n)
    assert tuple(route) == want
    for x, y in zip(both, got):
        np.testing.assert_allclose(x[0], y, rtol=0, atol=1e-15)
    ref = compat.polish_peaks_with_weights(A, B, data.gamma, w, half, 2)
    ref1 = path1.polish_single_peak(A, B, data.gamma, w, n, half, 2)
    for res, r in ((got, ref), (one, ref1)):
        for g, x, tol in zip(res, r, (3e-13, 3e-11, 1e-12)):
            np.testing.assert_allclose(g, x, rtol=0, atol=tol)
