"""A batch of windows runs as many rounds as the window with the most trials."""

import numpy as np
import pytest

from g2o_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("iterations,far", [(1, False), (2, False), (6, False), (7, True), (12, True)])
def test_rounds_are_the_most_trials(iterations, far):
    from g2o_b200 import backend
    windows = [synth.bundle_adjustment(5 + i, 150 + 20 * i, seed=60 + i) for i in range(5)]
    prm = backend.OptimizationAlgorithmFactory.instance().construct("lm_cuda")
    if far:  # trials are rejected on the way
        prm.initial_lambda = 1e-9
        rng = np.random.default_rng(4)
        for w in windows[1:3]:
            w.point_estimate += rng.normal(0.0, 3.0, w.point_estimate.shape)
    c = backend.CudaWindows(windows, prm)
    stats = c.optimize(iterations)
    most = max(s["trials"] for s in stats)
    assert stats[0]["rounds"] == most
    assert most >= iterations and (not far or most > iterations)
