"""Offset scans and polishes on cell moments (csrc/k2_cells.cu) at the edges of their tiles and cells,
against forms that do not use them: point evaluations by the plain kernel for the scans, the polishes
on exact A/B matrices for the polishes.

Tolerances.  A moment term carries the phasor's rounding (4e-16), the series' first dropped term (at most
1e-15) and the sums' roundings, per unit of sum 2|c| w (about 1.5 on these tables), against the plain
kernel's 2e-13: 3e-13 for a scan.  A polish's offset may differ by the sensitivity limit, 1e-10 of the
step clamp 1e-4, or by the order of the sums amplified along the path (bounded here by 1e-12); h then
by |h'| <= sum 2|c| w gamma < 3e3 times 1e-14.
"""
import math

import numpy as np
import pytest

from mertens_bound_b200 import compat, k2, path1, synth
from mertens_bound_b200._lib import check, lib, ptr

pytestmark = pytest.mark.gpu

N = 9000


@pytest.fixture(scope="module")
def setup(gpu):
    data = synth.make_table(N, seed=81)
    t = k2.ZeroTable.from_data(data)
    yield data, t
    t.close()


def _points(c, step, m0, n_m):
    base = [(int(a) << 64) | int(b) for a, b in zip(c.v_int, c.v_frac)]
    v = [(b + (m0 + m) * step) for b in base for m in range(n_m)]
    return synth.Candidates(np.array([x >> 64 for x in v], np.uint64),
                            np.array([x & (2**64 - 1) for x in v], np.uint64), np.zeros(len(v)))


# steps in 2^-64: 5e-7, 1.5e-4, 0.01 (few cells, many cells, the direct kernel's) and 3 + 2^-64
STEPS = [int(5e-7 * 2**64), int(1.5e-4 * 2**64), int(0.01 * 2**64), (3 << 64) + 1]


@pytest.mark.parametrize("P,n,m0,n_m", [(1, 1, -1, 2), (1, 9000, -120, 241), (3, 40, 0, 33), (8, 255, -500, 77),
                                        (9, 300, 7, 64), (64, 256, -38, 77), (65, 4097, -128, 257), (130, 777, -16, 33)])
@pytest.mark.parametrize("step", STEPS)
def test_hit_scan_edges(setup, P, n, m0, n_m, step):
    data, t = setup
    c = synth.make_candidates(P, seed=P + n_m)
    h = np.empty((P, n_m))
    check(lib().mb_hit_scan(t.handle, P, ptr(c.v_int), ptr(c.v_frac), 3e-9, n, step >> 64, step & (2**64 - 1), m0,
                            n_m, ptr(h)))
    T = data.gamma[n] if n < N else math.inf
    val, _, _ = k2.k2_plain(t, _points(c, step, m0, n_m), 3e-9, T)
    assert np.max(np.abs(h.reshape(-1) - val)) < 3e-13


@pytest.mark.parametrize("n_m", [31, 200, 4097])
@pytest.mark.parametrize("step", STEPS)
def test_grid_scan_edges(setup, n_m, step):
    """Two base points, one at the end of the 64.64 range, where a block's middle point would wrap."""
    data, t = setup
    c = synth.make_candidates(2, seed=n_m)
    c.v_int[1], c.v_frac[1] = 0, 12345
    h = np.empty((2, n_m))
    check(lib().mb_grid_scan(t.handle, 2, ptr(c.v_int), ptr(c.v_frac), 3e-9, 5000.0, step >> 64,
                             step & (2**64 - 1), 0, n_m, ptr(h)))
    val, _, _ = k2.k2_plain(t, _points(c, step, 0, n_m), 3e-9, 5000.0)
    assert np.max(np.abs(h.reshape(-1) - val)) < 3e-13
    c.v_int[1], c.v_frac[1] = 2**64 - 1, 2**64 - 1          # the grid leaves the range: the direct kernel
    check(lib().mb_grid_scan(t.handle, 2, ptr(c.v_int), ptr(c.v_frac), 3e-9, 5000.0, step >> 64,
                             step & (2**64 - 1), -1, 2, ptr(h)))
    assert np.all(np.isfinite(h[:, :1]))


def _weights(data, k):
    g = data.gamma
    u = g / g[-1]
    return [(1.0 - u) * np.cos(np.pi * u) + np.sin(np.pi * u) / np.pi, np.exp(-3e-9 * g * g), np.ones_like(g),
            np.where(np.arange(N) < 50, 1.0, 0.0), np.sin(g), -np.exp(-1e-7 * g * g)][:k]


def _close(got, want):
    for g, w, tol in zip(got, want, (3e-13, 3e-11, 1e-12)):
        np.testing.assert_allclose(g, w, rtol=0, atol=tol)


@pytest.mark.parametrize("P,n,W,half", [(1, 5, 1, 2.5e-4), (9, 63, 2, 2.5e-4), (70, 4096, 3, 2.5e-4),
                                        (64, 4097, 4, 2.5e-4), (5, 9000, 6, 2.5e-4), (3, 9000, 5, 0.0),
                                        (2, 2000, 2, 0.6)])
def test_polish_weights_edges(setup, P, n, W, half):
    """n below, at and above the 4,096 zeros of the grid stage; one to six weight vectors (two moment
    passes); a grid so wide that the cells give way to the A/B matrices."""
    data, t = setup
    c = synth.make_candidates(P, seed=90 + P)
    c.delta[:] = np.random.default_rng(P).uniform(-1e-4, 1e-4, P)
    ws = _weights(data, W)
    slots = [t.add_weights(w) for w in ws]
    hu, hp, dp = path1.polish_peaks_weights(t, c, slots, n, half, 40)
    A, B = path1.compute_exact_AB(t, c, n)
    for i, w in enumerate(ws):
        _close((hu[i], hp[i], dp[i]), compat.polish_peaks_with_weights(A, B, data.gamma[:n], w[:n], half, 40))


@pytest.mark.parametrize("P,n,steps", [(1, 7, 40), (8, 500, 0), (66, 9000, 40)])
def test_polish_single_edges(setup, P, n, steps):
    data, t = setup
    c = synth.make_candidates(P, seed=100 + P)
    w = _weights(data, 1)[0]
    got = path1.polish_single_exact(t, c, t.add_weights(w), n, 4e-5, steps)
    A, B = path1.compute_exact_AB(t, c, n)
    _close(got, path1.polish_single_peak(A, B, data.gamma[:n], w[:n], n, 4e-5, steps))


@pytest.mark.parametrize("P,n,top", [(1, 3, 1), (7, 511, 3), (65, 513, 65), (70, 9000, 25)])
def test_taylor_polish_edges(setup, P, n, top):
    data, t = setup
    c = synth.make_candidates(P, seed=110 + P)
    c.delta[:] = np.random.default_rng(P).uniform(-1e-4, 1e-4, P)
    w = _weights(data, 1)[0]
    got = path1.fast_polish_exact(t, c, t.add_weights(w), n, top=top)
    A, B = path1.compute_exact_AB(t, c, n)
    _close(got, path1.fast_polish_batch(A, B, data.gamma[:n], w[:n], top=top))


def test_sensitive_paths_take_the_direct_loops(gpu):
    """Under a weight vector without decay, Newton's six clamped steps amplify rounding by up to 1e9 on
    some peaks; those are polished by the loops over the zeros, so every offset agrees with the matrix
    form although the paths do not converge."""
    data = synth.make_table(60_000, seed=1)
    c = synth.make_candidates(96, seed=120)
    with k2.ZeroTable.from_data(data) as t:
        w = np.ones(data.n)
        got = path1.polish_peaks_exact(t, c, t.add_weights(w))
        A, B = path1.compute_exact_AB(t, c)
        want = compat.polish_peaks_with_weights(A, B, data.gamma, w, 2.5e-4, 40)
    np.testing.assert_allclose(got[0], want[0], rtol=0, atol=3e-13)
    np.testing.assert_allclose(got[2], want[2], rtol=0, atol=1e-12)
    # |h'| <= sum 2|c| gamma ~ 1.5e4 at an offset that does not converge
    np.testing.assert_allclose(got[1], want[1], rtol=0, atol=1.5e-10)
