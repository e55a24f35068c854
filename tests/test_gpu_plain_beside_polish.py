"""mb_k2_plain_dev in flight on the caller's stream keeps its partial sums in the table; a polish or a scan on cell moments
called meanwhile (on the table's own stream) does not touch them."""
import numpy as np
import pytest

from mertens_bound_b200 import hit_polish, k2, path1, synth
from mertens_bound_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def test_plain_in_flight(gpu):
    import torch
    n, P = 200_000, 4096
    data = synth.make_table(n, seed=101)
    c = synth.make_candidates(P, seed=102)
    few = c.subset(np.arange(256))
    pts = hit_polish.points_from_x(synth.leaves_x(64, 3))
    dev = torch.device("cuda", 0)
    vi, vf = (torch.from_numpy(a.view(np.int64).copy()).to(dev) for a in (c.v_int, c.v_frac))
    delta = torch.zeros(P, dtype=torch.float64, device=dev)
    out = torch.empty(3, P, dtype=torch.float64, device=dev)
    stream = torch.cuda.Stream(dev)
    torch.cuda.synchronize(dev)
    with k2.ZeroTable.from_data(data) as t:
        s = t.add_weights(np.exp(-3e-9 * data.gamma**2))

        def plain():
            out.zero_()
            torch.cuda.synchronize(dev)
            check(lib().mb_k2_plain_dev(t.handle, P, vi.data_ptr(), vf.data_ptr(), delta.data_ptr(), 3e-9,
                                        float("inf"), out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(),
                                        stream.cuda_stream))

        def calls():
            return [*path1.polish_peaks_exact(t, few, s), *path1.polish_single_exact(t, few, s),
                    *path1.fast_polish_exact(t, few, s), hit_polish.polish_hits(t, pts, thresholds=(None,) * 3).h]

        plain()
        stream.synchronize()
        want, alone = out.cpu().numpy(), calls()
        for _ in range(3):
            plain()                                    # ~3 ms on the GPU
            got = calls()
            stream.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)
            assert all(np.array_equal(x, y) for x, y in zip(got, alone))
