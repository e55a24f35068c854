"""The Taylor polish's grid stage gives a peak the same bits whatever the peaks beside it: one peak group per warp, tiles of
128 peaks and passes of at most 256 MB of sums are all the same to it."""
import numpy as np
import pytest

from mertens_bound_b200 import k2, path1, score, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 10_000, 100_000])
def test_grid_stage_does_not_depend_on_the_batch(gpu, n):
    data = synth.make_table(100_000, seed=82).truncate(n)
    P = 6000                                # two passes at 100,000 zeros: 297 chunks x 24 sums x 8 bytes a peak
    c = synth.make_candidates(P, seed=83)
    c.delta[:] = np.random.default_rng(83).uniform(-1e-4, 1e-4, P)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(score.reference_weights(data.gamma)["jp"])
        want = path1.fast_polish_exact(t, c, s, top=0)
        for rows in (np.arange(1), np.arange(7), np.arange(9, 40), np.arange(100, 1200), np.arange(4500, 4900)):
            got = path1.fast_polish_exact(t, c.subset(rows), s, top=0)
            assert all(np.array_equal(g, w[rows]) for g, w in zip(got, want))
