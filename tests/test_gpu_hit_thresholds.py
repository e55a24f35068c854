"""Thresholds of the staged hit polish at their edges: lists shorter than the three stages that have one, and |h| that is
not a number."""
import math

import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, synth

pytestmark = pytest.mark.gpu


def _points(P):
    return hit_polish.points_from_x(synth.leaves_x(P, 7))


def test_short_threshold_lists(gpu):
    data = synth.make_table(3000, seed=43)
    pts = _points(5)
    with k2.ZeroTable.from_data(data) as t:
        full = hit_polish.polish_hits(t, pts, thresholds=(None, math.inf, None))
        for thr in ((), (None,), (0.0,), (None, None), (0.0, -math.inf)):       # a hit needs the missing entry
            with pytest.raises(IndexError):
                hit_polish.polish_hits(t, pts, thresholds=thr)
        dead = hit_polish.polish_hits(t, pts, thresholds=(math.inf,))           # none does
        assert np.all(dead.stage == 0) and np.all(dead.h != 0.0)
        dead = hit_polish.polish_hits(t, pts, thresholds=(None, math.inf))
        for f in ("h", "dy", "stage"):
            assert np.array_equal(getattr(dead, f), getattr(full, f))
        assert len(hit_polish.polish_hits(t, pts[:0], thresholds=()).h) == 0


def test_overflowing_sums(gpu):
    """Coefficients whose sums overflow: h is infinite or NaN.  Without thresholds every hit runs all stages; a NaN
    passes no threshold of the caller's, -inf included."""
    data = synth.make_table(3000, seed=43)
    data.c_re[:256] = 1.7e308
    data.c_im[:256] = 0.0
    pts = _points(5)
    with k2.ZeroTable.from_data(data) as t:
        r = hit_polish.polish_hits(t, pts, k=0.0, thresholds=(None, None, None))
        assert np.all(np.isnan(r.h)) and np.all(r.stage == 4)
        # the first point wherever all are NaN
        want = -sum(m * hit_polish._fixed(st) for _, m, st, _, _ in hit_polish.STAGES[1:]) / 2.0**64
        np.testing.assert_allclose(r.dy, want, rtol=1e-15)
        for thr in (-math.inf, 0.0, math.nan):
            r = hit_polish.polish_hits(t, pts, k=0.0, thresholds=(thr, None, None))
            assert np.all(r.stage == 0)
