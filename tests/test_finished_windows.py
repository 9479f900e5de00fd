"""A finished window keeps its estimates, bit for bit, in the rounds that other
windows of its batch need."""

import numpy as np
import pytest

from g2o_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("iterations", [7, 12])
def test_same_bits_alone_and_beside_a_slow_window(iterations):
    from g2o_b200 import backend
    windows = [synth.bundle_adjustment(5 + i, 150 + 20 * i, seed=60 + i) for i in range(5)]
    prm = backend.OptimizationAlgorithmFactory.instance().construct("lm_cuda")
    prm.initial_lambda = 1e-9  # trials are rejected on the way
    rng = np.random.default_rng(4)
    for w in windows[1:3]:
        w.point_estimate += rng.normal(0.0, 3.0, w.point_estimate.shape)
    c = backend.CudaWindows(windows, prm)
    stats = c.optimize(iterations)
    assert max(s["trials"] for s in stats) > min(s["trials"] for s in stats)
    for i, w in enumerate(windows):
        a = backend.CudaWindows([w], prm)
        s = a.optimize(iterations)[0]
        assert (s["trials"], s["iterations"]) == (stats[i]["trials"], stats[i]["iterations"])
        assert all(np.array_equal(x, y) for x, y in zip(a.estimates(0), c.estimates(i)))
