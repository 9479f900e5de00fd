"""Waits of the tiled Cholesky that run out (a flag that nothing sets): every
solve reports them, and the call after a reported one works."""

import numpy as np
import pytest

from g2o_b200 import synth


def problem(monkeypatch, kind, solver="gn_cuda_chol_mixed"):
    from g2o_b200 import backend
    g = synth.pose_graph_2d(60, 30, seed=2)
    if kind:
        monkeypatch.setenv("G2OC_TEST_BARRIER_EXTRA", kind)
    p = backend.CudaProblem(g, backend.OptimizationAlgorithmFactory.instance().construct(solver))
    monkeypatch.delenv("G2OC_TEST_BARRIER_EXTRA", raising=False)
    return p


def timed_out(call):
    from g2o_b200 import backend
    from g2o_b200.abi import G2OC_ERR_TIMEOUT
    with pytest.raises(backend.G2ocError) as e:
        call()
    return e.value.status == G2OC_ERR_TIMEOUT


# the outcome read by the host before a refinement, and at the end of the trial
@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["gn_cuda_chol_mixed", "gn_cuda", "lm_cuda_chol_mixed"])
def test_call_after_a_timeout(monkeypatch, solver):
    p = problem(monkeypatch, "2", solver)
    start = p.estimates()[0]
    assert timed_out(lambda: p.optimize(1))
    p.set_estimates(start)
    good = problem(monkeypatch, None, solver)
    done, stats = p.optimize(3)
    assert done == good.optimize(3)[0] == 3
    assert np.array_equal(p.estimates()[0], good.estimates()[0])


@pytest.mark.gpu
def test_timeout_of_a_correction(monkeypatch):
    p = problem(monkeypatch, "3")
    assert timed_out(lambda: p.optimize(1))
