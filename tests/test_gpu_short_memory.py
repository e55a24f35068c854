"""Scans and polishes on a device with little free memory: where the cell moments do not fit, the calls take the loops over
the zeros, which need no workspace, as before there were moments.  Results agree as closely as the two ways do
(test_gpu_cells.py)."""
import ctypes as C

import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, path1, synth
from mertens_bound_b200._lib import check, lib, ptr

pytestmark = pytest.mark.gpu

N, FREE = 20_000, 40 << 20


def _redone(table):
    n = C.c_int64()
    check(lib().mb_table_polish_redone(table.handle, C.byref(n)))
    return n.value


def _calls(t, slots, c, pts, half):
    few = c.subset(np.arange(300))
    step = hit_polish._fixed(1.5e-4)
    h = np.empty((c.n, 241))

    def scan():
        check(lib().mb_hit_scan(t.handle, c.n, ptr(c.v_int), ptr(c.v_frac), 3e-9, N, 0, step, -120, 241, ptr(h)))
        return (h.copy(),)

    def polish():
        r = hit_polish.polish_hits(t, pts, thresholds=(None,) * 3)
        return r.h, r.dy

    return [lambda: path1.polish_peaks_weights(t, few, slots, None, half, 40),
            lambda: path1.polish_peaks_exact(t, c, slots[0], None, half, 40),
            lambda: path1.polish_single_exact(t, c, slots[0], None, half, 10),
            lambda: path1.fast_polish_exact(t, c, slots[0], None, np.linspace(-half, half, 41), top=c.n), scan, polish]


def test_calls_with_little_free_memory(gpu):
    import torch
    data = synth.make_table(N, seed=96)
    g = data.gamma
    ws = [np.exp(-3e-9 * g * g), np.exp(-1e-8 * g * g), np.exp(-2e-8 * g * g), np.exp(-4e-8 * g * g),
          np.exp(-8e-8 * g * g)]
    c = synth.make_candidates(1024, seed=97)
    pts = hit_polish.points_from_x(synth.leaves_x(600, 98))
    with k2.ZeroTable.from_data(data) as t:
        slots = [t.add_weights(w) for w in ws]
        want = [f() for f in _calls(t, slots, c, pts, 2.5e-4)]
        assert _redone(t) >= 0
        for f in _calls(t, slots, c, pts, 0.3):                # the loops over the zeros, loaded
            f()
    with k2.ZeroTable.from_data(data) as t:
        slots = [t.add_weights(w) for w in ws]
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - FREE, dtype=torch.uint8, device="cuda")
        try:
            got, routes = [], []
            for f in _calls(t, slots, c, pts, 2.5e-4):
                got.append(f())
                routes.append(_redone(t))
        finally:
            del fill
            torch.cuda.empty_cache()
        assert routes[:4] == [-1] * 4
        again = [f() for f in _calls(t, slots, c, pts, 2.5e-4)]
        assert _redone(t) >= 0
    for a, b in zip(again, want):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    for i, (a, b) in enumerate(zip(got, want)):
        for x, y, tol in zip(a, b, (3e-13, 3e-11, 1e-12) if i < 4 else (1e-11, 1e-12)):
            np.testing.assert_allclose(x, y, rtol=0, atol=tol)
