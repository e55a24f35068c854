"""The second pass of the polishes on cell moments (csrc/k2_cells.cu): peaks whose Newton path amplifies rounding are
polished again over the zeros, in batches of at most 256 MB of (A, B), each pass by 64 CTAs per peak.

Such peaks are rare (a few of 4,096 candidates), so the tests look for them and repeat them until their CTAs are many
times the GPU's slots and their batches several.  Each copy has to give the same bits, and those of the matrix form
within 1e-12 in the offset (the second pass adds the matrix form's terms in its order) and that times
sum 2|c| w gamma >= |h'| in h."""
import ctypes as C

import numpy as np
import pytest

from mertens_bound_b200 import compat, k2, path1, synth
from mertens_bound_b200._lib import check, lib

pytestmark = pytest.mark.gpu

N = 200_000
BATCH = (256 << 20) // (16 * N)          # 83 peaks


def redone(table):
    n = C.c_int64()
    check(lib().mb_table_polish_redone(table.handle, C.byref(n)))
    return n.value


def find(table, polish, c, rows):
    """The rows of c whose polish takes the second pass, by halving."""
    polish(table, c.subset(rows))
    k = redone(table)
    if k == 0:
        return []
    if k == len(rows):
        return list(rows)
    h = len(rows) // 2
    return find(table, polish, c, rows[:h]) + find(table, polish, c, rows[h:])


@pytest.mark.parametrize("mode", ["peaks", "single"])
def test_many_sensitive_peaks(gpu, mode):
    data = synth.make_table(N, seed=1)
    g = data.gamma
    w = g / g[-1]
    c = synth.make_candidates(4096, seed=120)
    with k2.ZeroTable.from_data(data) as t:
        slot = t.add_weights(w)

        def polish(table, cands):
            if mode == "peaks":
                return path1.polish_peaks_exact(table, cands, slot)
            return path1.polish_single_exact(table, cands, slot, N, 4e-5, 40)

        rows = np.array(find(t, polish, c, np.arange(c.n)))
        assert 1 <= len(rows) <= 64
        other = np.setdiff1d(np.arange(40), rows)
        idx = np.concatenate([np.tile(rows, -(-4 * BATCH // len(rows))), other])
        np.random.default_rng(3).shuffle(idx)
        many = c.subset(idx)
        got = polish(t, many)
        assert redone(t) == len(idx) - len(other) >= 4 * BATCH
        for _ in range(4):
            again = polish(t, many)
            assert all(np.array_equal(a, b) for a, b in zip(got, again))
        for r in rows:
            at = np.flatnonzero(idx == r)
            assert all(np.all(x[at] == x[at[0]]) for x in got)
        uniq = np.concatenate([rows, other])
        A, B = path1.compute_exact_AB(t, c.subset(uniq))
    if mode == "peaks":
        want = compat.polish_peaks_with_weights(A, B, g, w, 2.5e-4, 40)
    else:
        want = path1.polish_single_peak(A, B, g, w, N, 4e-5, 40)
    first = np.array([np.flatnonzero(idx == r)[0] for r in uniq])
    slope = np.sum(2.0 * np.hypot(data.c_re, data.c_im) * w * g)
    scale = np.sum(2.0 * np.hypot(data.c_re, data.c_im) * w)
    np.testing.assert_allclose(got[0][first], want[0], rtol=0, atol=1e-13 * scale)
    np.testing.assert_allclose(got[2][first], want[2], rtol=0, atol=1e-12)
    np.testing.assert_allclose(got[1][first], want[1], rtol=0, atol=1e-12 * slope)


def test_second_pass_of_several_weights(gpu):
    """Six vectors (two moment passes), each list in its own batches; the rows equal the single-vector calls."""
    data = synth.make_table(N, seed=1)
    g = data.gamma
    u = g / g[-1]
    c = synth.make_candidates(4096, seed=120)
    with k2.ZeroTable.from_data(data) as t:
        slots = [t.add_weights(w) for w in (u, np.exp(-1e-10 * g * g), u * u, (u > 0.5) * 1.0, np.sin(g), 1.0 - u)]
        rows = np.array(find(t, lambda tb, x: path1.polish_peaks_exact(tb, x, slots[0]), c, np.arange(c.n)))
        many = c.subset(np.concatenate([np.tile(rows, -(-2 * BATCH // len(rows))), np.arange(30)]))
        got = path1.polish_peaks_weights(t, many, slots)
        total = redone(t)
        assert total >= 2 * BATCH
        one = 0
        for i, s in enumerate(slots):
            want = path1.polish_peaks_exact(t, many, s)
            one += redone(t)
            assert all(np.array_equal(x[i], y) for x, y in zip(got, want))
        assert one == total


@pytest.mark.parametrize("steps", [10, 40])
def test_starts_that_end_near_one_maximum(gpu, steps):
    """The single-peak loop's two starts can end within rounding of the same |h| at offsets 1e-13 to 1e-11 apart; which one
    is kept then follows from the loops' own rounding, so the second pass decides.  The offsets of all peaks agree with
    the matrix form's to twice the loop's last step, 1e-14."""
    data = synth.make_table(20_000, seed=96)
    w = np.exp(-3e-9 * data.gamma**2)
    c = synth.make_candidates(1024, seed=97)
    with k2.ZeroTable.from_data(data) as t:
        got = path1.polish_single_exact(t, c, t.add_weights(w), None, 2.5e-4, steps)
        n = redone(t)
        A, B = path1.compute_exact_AB(t, c)
    want = path1.polish_single_peak(A, B, data.gamma, w, data.n, 2.5e-4, steps)
    assert 4 <= n <= 100
    np.testing.assert_allclose(got[2], want[2], rtol=0, atol=2e-14)
    np.testing.assert_allclose(got[1], want[1], rtol=0, atol=1e-14)
