"""The windows' dense systems as one batch of tiles: windows whose unknowns end
on, before and after a tile of 64, windows without free cameras, and windows
that finish at different rounds give what each gives alone."""

import numpy as np
import pytest

from g2o_b200 import synth


def window(cams, points, seed):
    g = synth.bundle_adjustment(cams, points, seed=seed)
    return g


# free cameras of the windows (two are fixed): n = 6 (cams - 2) around 64 and 128
@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[3], [12, 13], [2, 5, 12], [23, 24, 2, 34], [13, 60, 4, 12, 45, 3]])
def test_batch_matches_windows_alone(sizes):
    from g2o_b200 import backend
    prm = backend.OptimizationAlgorithmFactory.instance().construct("lm_cuda")
    ws = [window(c, 40 + 9 * c, 70 + i) for i, c in enumerate(sizes)]
    both = backend.CudaWindows(ws, prm)
    stats = both.optimize(4)
    for i, g in enumerate(ws):
        one = backend.CudaWindows([g], prm)
        s = one.optimize(4)[0]
        assert (s["iterations"], s["trials"], s["solve_ok"]) == (stats[i]["iterations"], stats[i]["trials"],
                                                                 stats[i]["solve_ok"])
        assert s["chi2"] == stats[i]["chi2"]  # a window's sums do not depend on the others
        assert all(np.array_equal(a, b) for a, b in zip(both.estimates(i), one.estimates(0)))
