"""A leaf's screen scores and its decisions do not depend on the leaves that it is screened with: the same bits with one
and four leaves per thread, and on both walks of the survivors' list (a leaf per thread, eight lanes per leaf)."""
import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, synth

pytestmark = pytest.mark.gpu

FOUR = 148 * 4 * 256          # leaves from which a 148-SM device screens four per thread


@pytest.mark.parametrize("high", [False, True])               # both records: gamma below and above 3.29e6
@pytest.mark.parametrize("ends", [(64, 128, 256), (5, 13, 14, 1024), (1, 2, 3, 4, 5, 6, 7, 8)])
def test_scores_do_not_depend_on_the_batch(gpu, small_table, high, ends):
    data = small_table
    if high:
        rng = np.random.default_rng(91)
        gam = 5.0e6 + np.cumsum(rng.uniform(0.2, 0.72, 3000))
        G3 = synth.fixed_from_double(gam / (2.0 * np.pi), rng)
        data = synth.ZeroTableData(G3, synth.gamma_from_fixed(G3), data.c_re[:3000].copy(), data.c_im[:3000].copy(),
                                   data.seed)
    k = 0.0 if high else 3e-9
    c = synth.make_candidates(FOUR + 999, seed=19)
    pts = np.stack([c.v_int, c.v_frac], axis=1).astype(np.uint64)
    with k2.ZeroTable.from_data(data) as t:
        def run(p, thr):
            return hit_polish.screen_leaves(t, p, k, (ends, thr), max_hits=len(p), all_scores=True)

        every = run(pts, (-1.0,) * len(ends)).scores              # a leaf per thread throughout
        thr = tuple(float(np.quantile(every[:, s], 0.9)) for s in range(len(ends)))
        alive = np.cumprod(every >= np.array(thr, np.float32), axis=1).astype(bool)
        want = every.copy()
        want[:, 1:][~alive[:, :-1]] = -1.0
        hits = np.flatnonzero(alive[:, -1])
        few = run(pts, thr)                                       # a tenth goes on: eight lanes per leaf
        assert np.array_equal(few.scores, want) and np.array_equal(few.hits, hits)
        on = np.flatnonzero(alive[:, 0])
        for rows in (on[:700], on[:65], on[:1], np.arange(513), np.concatenate([on[:3], np.arange(300)])):
            part = run(pts[rows], thr)                            # batches that all or hardly any pass
            assert np.array_equal(part.scores, want[rows])
            assert np.array_equal(part.hits, np.flatnonzero(alive[rows, -1]))
