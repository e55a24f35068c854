"""Calls of more points than one pass takes: peak chunks of the polishes on cell moments, base-point chunks of the scans on
them, peak chunks of the A/B matrices (moments and matrices are held to 256 MB and 4 GiB a pass)."""
import ctypes as C

import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, path1, synth
from mertens_bound_b200._lib import check, lib, ptr

pytestmark = pytest.mark.gpu


def _redone(table):
    n = C.c_int64()
    check(lib().mb_table_polish_redone(table.handle, C.byref(n)))
    return n.value


def test_polish_peak_chunks(gpu):
    """About 600 cells x 176 bytes x 5 vectors a peak: some 500 peaks a chunk, so 1,300 take three.  A peak's results have
    the bits of a call without the others."""
    data = synth.make_table(20_000, seed=96)
    g = data.gamma
    c = synth.make_candidates(1300, seed=99)
    c.delta[:] = np.random.default_rng(99).uniform(-1e-4, 1e-4, c.n)
    with k2.ZeroTable.from_data(data) as t:
        slots = [t.add_weights(np.exp(-k * g * g)) for k in (3e-9, 1e-9, 1e-8, 2e-8, 4e-8, 8e-8)]
        got = path1.polish_peaks_weights(t, c, slots)
        assert _redone(t) >= 0
        top = path1.fast_polish_exact(t, c, slots[0], top=c.n)
        for rows in (np.arange(40), np.arange(480, 560), np.arange(1000, 1060), np.arange(1260, 1300)):
            part = path1.polish_peaks_weights(t, c.subset(rows), slots)
            assert all(np.array_equal(p, x[:, rows]) for p, x in zip(part, got))
            part = path1.fast_polish_exact(t, c.subset(rows), slots[0], top=len(rows))
            assert all(np.array_equal(p, x[rows]) for p, x in zip(part, top))


@pytest.mark.parametrize("n,step,n_m", [(20_000, 5e-7, 241), (512, 2.5e-5, 457)])
def test_scan_base_point_chunks(gpu, n, step, n_m):
    """70,000 base points: more blocks than a grid dimension takes (65,535).  3e-13 as in test_gpu_cells.py."""
    data = synth.make_table(20_000, seed=96)
    P, m0, st = 70_000, -(n_m // 2), hit_polish._fixed(step)
    c = synth.make_candidates(P, seed=100)
    h = np.empty((P, n_m))
    rows = np.unique(np.concatenate([np.linspace(0, P - 1, 60).astype(int), np.arange(65530, 65540)]))
    base = [(int(c.v_int[p]) << 64 | int(c.v_frac[p])) for p in rows]
    v = [b + (m0 + m) * st for b in base for m in range(n_m)]
    pts = synth.Candidates(np.array([x >> 64 for x in v], np.uint64),
                           np.array([x & (2**64 - 1) for x in v], np.uint64), np.zeros(len(v)))
    with k2.ZeroTable.from_data(data) as t:
        check(lib().mb_hit_scan(t.handle, P, ptr(c.v_int), ptr(c.v_frac), 3e-9, n, 0, st, m0, n_m, ptr(h)))
        val, _, _ = k2.k2_plain(t, pts, 3e-9, float(data.gamma[n]) if n < data.n else float("inf"))
    assert np.max(np.abs(h[rows].reshape(-1) - val)) < 3e-13


def test_matrix_peak_chunks(gpu):
    """A grid too wide for the cells on 600,000 zeros: the 4 GiB of A/B matrices hold 447 peaks, so 460 take two chunks."""
    data = synth.make_table(600_000, seed=72)
    c = synth.make_candidates(460, seed=73)
    c.delta[:] = np.random.default_rng(73).uniform(-1e-4, 1e-4, c.n)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(np.exp(-3e-9 * data.gamma**2))
        got = path1.polish_peaks_weights(t, c, [s], None, 0.08, 3)
        assert _redone(t) == -1
        want = path1.polish_peaks_exact(t, c, s, None, 0.08, 3)
        assert _redone(t) == -1
    for x, y in zip(got, want):
        np.testing.assert_allclose(x[0], y, rtol=0, atol=1e-15)
