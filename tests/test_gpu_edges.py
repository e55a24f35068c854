"""Kernel variants at the sizes where their rules change over: four leaves per thread in the screen (and
its split records above gamma = 3.29e6), the plain kernel's tile widths, the heavy tier's groups of at most 32
candidates, the certified kernel's tiles of four candidates, 16-term scans over one and two peak groups per warp, and the hit polish's early exits.
Tolerances are those of the general tests of each path: 2e-5 for a screen score (MUFU and FP32 sums), 2e-13 for
the plain kernel and 3e-13 for a scan against it, a plan's own bounds for the tiers."""
import math

import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, synth
from mertens_bound_b200._lib import check, lib, ptr
from oracle.oracle import Oracle, reference_format, zerodata_polish

pytestmark = pytest.mark.gpu

SCORE_TOL = 2e-5
FOUR = 148 * 4 * 256          # leaves from which a 148-SM device screens four per thread


@pytest.fixture(scope="module")
def table(gpu, small_table):
    t = k2.ZeroTable.from_data(small_table)
    yield t
    t.close()


@pytest.fixture(scope="module")
def high(gpu, small_table):
    """3,000 zeros above gamma = 5e6."""
    rng = np.random.default_rng(91)
    gam = 5.0e6 + np.cumsum(rng.uniform(0.2, 0.72, 3000))
    G3 = synth.fixed_from_double(gam / (2.0 * math.pi), rng)
    data = synth.ZeroTableData(G3, synth.gamma_from_fixed(G3), small_table.c_re[:3000].copy(),
                               small_table.c_im[:3000].copy(), small_table.seed)
    t = k2.ZeroTable.from_data(data)
    yield data, t
    t.close()


def _stage_scores(oracle, data, pts, k, ends, step):
    st = hit_polish._fixed(step)
    best = np.zeros((len(pts), len(ends)))
    for m in range(-3, 4):
        v = [(int(a) << 64 | int(b)) + m * st for a, b in pts]
        c = synth.Candidates(np.array([x >> 64 for x in v], np.uint64),
                             np.array([x & (2**64 - 1) for x in v], np.uint64), np.zeros(len(v)))
        for s, e in enumerate(ends):
            best[:, s] = np.maximum(best[:, s], np.abs(oracle.k2(c, data, k, e)[0][:, 0]))
    return best


@pytest.mark.parametrize("P", [1, 257, FOUR - 1, FOUR, FOUR + 1, 2 * FOUR + 777])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("share", [0.6, 0.04])       # of the leaves alive after a stage: both list walks
def test_screen_leaves_per_thread(table, small_table, high, oracle, P, split, share):
    data, t = high if split else (small_table, table)
    k = 0.0 if split else 3e-9
    c = synth.make_candidates(P, seed=17)
    pts = np.stack([c.v_int, c.v_frac], axis=1).astype(np.uint64)
    ends, step = (64, 128, 256), hit_polish.SCREEN_STEP
    probe = hit_polish.screen_leaves(t, pts[:4096], k, (ends, (-1.0,) * 3), step, all_scores=True).scores
    thr = tuple(float(np.quantile(probe[:, s], 1.0 - share)) for s in range(3))
    r = hit_polish.screen_leaves(t, pts, k, (ends, thr), step, max_hits=P, all_scores=True)
    rows = np.unique(np.concatenate([np.arange(min(P, 24)), np.arange(max(0, P - 24), P)]))
    want = _stage_scores(oracle, data, pts[rows], k, ends, step)
    got = r.scores[rows]
    assert np.max(np.abs(got - want)[got >= 0]) <= SCORE_TOL
    thr32 = np.array(thr, np.float32)
    reached = r.scores >= 0
    assert reached[:, 0].all()
    for s in range(1, 3):
        assert np.array_equal(reached[:, s], np.all(r.scores[:, :s] >= thr32[:s], axis=1))
    assert np.array_equal(r.hits, np.flatnonzero(np.all(r.scores >= thr32, axis=1)))
    assert np.array_equal(r.hit_scores, r.scores[r.hits])


@pytest.mark.parametrize("P", [63, 65, 2047, 2048])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_plain_tile_edges(table, small_table, oracle, P, n):
    cd = synth.make_candidates(P, seed=P + n)
    cd.delta[:] = np.linspace(-3e-4, 3e-4, P)
    val, dd, dk = k2.k2_plain(table, cd, 1e-9, float(small_table.gamma[n]))
    rows = np.unique(np.linspace(0, P - 1, 40).astype(int))
    ohi, _ = oracle.k2(cd.subset(rows), small_table, 1e-9, n)
    for got, q in ((val, 0), (dd, 1), (dk, 2)):
        assert np.max(np.abs(got[rows] - ohi[:, q])) < 2e-13 * max(1.0, np.max(np.abs(ohi[:, q])))


@pytest.mark.parametrize("groups", [[1], [2, 31], [16], [32], [33], [32, 33, 1, 64]])
@pytest.mark.parametrize("n", [1, 63, 65, 10000])
def test_heavy_small_groups(table, small_table, oracle, groups, n):
    P = sum(groups)
    cd = synth.make_candidates(P, seed=P + n)
    cd.delta[:] = np.linspace(-3e-4, 3e-4, P)
    T = float(small_table.gamma[n]) if n < small_table.n else math.inf
    G = len(groups)
    with k2.Plan(table, groups, [3e-9] * G, [T] * G, tol=1e-14) as plan:
        gi = [plan.group_info(g) for g in range(G)]
        assert all(x["n_heavy"] == x["n_T"] == n for x in gi)
        got = plan.run(cd)
    ohi, _ = oracle.k2(cd, small_table, 3e-9, n)
    p = 0
    for g, nc in enumerate(groups):
        for q, key in ((0, "err_bound"), (1, "err_bound_dd"), (2, "err_bound_dk")):
            assert np.max(np.abs(got[q][p:p + nc] - ohi[p:p + nc, q])) <= gi[g][key]
        p += nc


@pytest.mark.parametrize("P", [63, 64, 65, 127, 129, 1023, 1025])
def test_scan_16_terms(table, small_table, P):
    """129 points of step 1.5e-4 over 900 zeros: 16-term cells where the peak count leaves the direct kernel."""
    n, step, m0, n_m = 900, int(1.5e-4 * 2**64), -64, 129
    c = synth.make_candidates(P, seed=P)
    h = np.empty((P, n_m))
    check(lib().mb_hit_scan(table.handle, P, ptr(c.v_int), ptr(c.v_frac), 3e-9, n, 0, step, m0, n_m, ptr(h)))
    rows = np.unique(np.linspace(0, P - 1, 70).astype(int))
    v = [(int(c.v_int[p]) << 64 | int(c.v_frac[p])) + (m0 + m) * step for p in rows for m in range(n_m)]
    pts = synth.Candidates(np.array([x >> 64 for x in v], np.uint64),
                           np.array([x & (2**64 - 1) for x in v], np.uint64), np.zeros(len(v)))
    val, _, _ = k2.k2_plain(table, pts, 3e-9, float(small_table.gamma[n]))
    assert np.max(np.abs(h[rows].reshape(-1) - val)) < 3e-13


@pytest.mark.parametrize("n,P", [(200, 1), (3000, 9), (10000, 24)])
def test_hit_polish_exits(gpu, n, P):
    """Thresholds at each stage's middle value: hits leave after every stage, the others go on."""
    data = synth.make_table(n, seed=43)
    rng = np.random.default_rng(n)
    xs = [int(rng.integers(3_400_000_000_000_000_000, 3_600_000_000_000_000_000)) << 30 |
          int(rng.integers(0, 1 << 30)) for _ in range(P)]
    pts = hit_polish.points_from_x(xs)
    with k2.ZeroTable.from_data(data) as t:
        thr, alive = [], np.ones(P, bool)
        for s in range(3):
            r = hit_polish.polish_hits(t, pts, thresholds=tuple(thr) + (math.inf,) + (None,) * (2 - s))
            b = np.sort(np.abs(r.h[alive]))
            thr.append(float((b[len(b) // 2 - 1] + b[len(b) // 2]) / 2) if len(b) > 1 else float(b[0]) * 0.5)
            assert np.all(r.stage[alive] == s)
            alive &= np.abs(r.h) >= thr[s]
        r = hit_polish.polish_hits(t, pts, thresholds=tuple(thr))
        empty = hit_polish.polish_hits(t, pts[:0])
    assert len(empty.h) == 0
    assert np.array_equal(r.stage == 4, alive)
    reft = reference_format(data, exact_psi=True)
    two_astar = 2 * reft["alpha"] * np.exp(-3e-9 * data.gamma ** 2)
    x_lo = np.array([x & ((1 << 64) - 1) for x in xs], np.uint64)
    x_hi = np.array([x >> 64 for x in xs], np.uint64)
    _, _, top = Oracle().ref_peak_AB((x_lo, x_hi, np.zeros(P)), reft, want_top=True)
    for i in range(P):
        h, dy = zerodata_polish(top[i].view(np.int64), two_astar, data.gamma, thresholds=tuple(thr))
        assert abs(r.h[i] - h) < 1e-11 * max(1.0, abs(h))
        assert abs(r.dy[i] - dy) < 1e-12


@pytest.mark.parametrize("P", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("n", [1, 257, 3000])
def test_certified_candidate_tiles(table, small_table, oracle, P, n):
    """Every interval holds the oracle's value; a radius per candidate widens its own interval alone."""
    cd = synth.make_candidates(P, seed=P + n)
    T = float(small_table.gamma[n])
    ohi, olo = oracle.k2(cd, small_table, 3e-9, n)
    lo, hi, ab = k2.k2_certified(table, cd, 3e-9, T)
    dlo, dhi = k2.k2_certified_grad(table, cd, 3e-9, T)
    rad = np.zeros(P)
    rad[P - 1] = 1e-9
    rlo, rhi, _ = k2.k2_certified(table, cd, 3e-9, T, v_rad=rad)
    # the FP64 oracle value and each end round by less than an ulp of the sum of amplitudes
    slack = 4e-16 * ab
    assert np.all(lo - slack <= ohi[:, 0]) and np.all(ohi[:, 0] <= hi + slack)
    assert np.all(hi - lo < 1e-13)
    assert np.array_equal(dlo[0], lo) and np.array_equal(dhi[0], hi)
    for row in (1, 2):
        eps = 4e-16 * np.abs(ohi[:, row])
        assert np.all(dlo[row] - eps <= ohi[:, row]) and np.all(ohi[:, row] <= dhi[row] + eps)
    wlo, whi = k2.k2_certified_grad(table, cd, 3e-9, T, k_hi=4e-9)           # a wide k: two exponentials
    mid = oracle.k2(cd, small_table, 3.5e-9, n)[0]
    for row in range(3):
        eps = 4e-16 * np.maximum(np.abs(mid[:, row]), ab)
        assert np.all(wlo[row] - eps <= mid[:, row]) and np.all(mid[:, row] <= whi[row] + eps)
    assert np.array_equal(rlo[:-1], lo[:-1]) and np.array_equal(rhi[:-1], hi[:-1])
    assert rlo[-1] < lo[-1] and rhi[-1] > hi[-1]


@pytest.mark.parametrize("half", [0.045, 0.055, 0.08])
def test_polish_cells_around_shared_memory(gpu, half):
    """About 1,060, 1,290 and 1,880 cells: the polish's moments fit shared memory (1,200 cells) or do not.  The
    matrix form's offsets agree to 1e-12 and h to 3e-11 (an offset of 1e-14 times |h'| < 3e3)."""
    from mertens_bound_b200 import compat, path1
    data = synth.make_table(9000, seed=81)
    c = synth.make_candidates(5, seed=95)
    w = np.exp(-3e-9 * data.gamma ** 2)
    with k2.ZeroTable.from_data(data) as t:
        got = path1.polish_peaks_exact(t, c, t.add_weights(w), None, half, 40)
        A, B = path1.compute_exact_AB(t, c)
    want = compat.polish_peaks_with_weights(A, B, data.gamma, w, half, 40)
    for g, x, tol in zip(got, want, (3e-13, 3e-11, 1e-12)):
        np.testing.assert_allclose(g, x, rtol=0, atol=tol)
