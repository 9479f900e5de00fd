"""An iteration whose every trial is rejected leaves the estimates as they were,
bit for bit: the update kernel saved them before each trial."""

import numpy as np
import pytest

from g2o_b200 import synth


def graph(kind):
    if kind == "2d":
        return synth.pose_graph_2d(300, 100, seed=5)
    if kind == "3d":
        return synth.pose_graph_3d(3, 40, seed=6)
    if kind == "stereo":
        return synth.stereo_bundle_adjustment(8, 400, seed=7)
    return synth.bundle_adjustment(8, 400, seed=9)


# information matrices of the other sign make H negative definite: no trial's
# factorization succeeds, and a failed one is a rejected one
@pytest.mark.gpu
@pytest.mark.parametrize("kind,solver", [("2d", "lm_cuda"), ("3d", "lm_cuda"), ("stereo", "lm_cuda_chol"),
                                         ("mono", "lm_cuda_chol"), ("2d", "lm_cuda_chol_mixed")])
def test_every_trial_rejected(kind, solver):
    from g2o_b200 import backend
    g = graph(kind)
    good = np.array(g.information)
    g.information = -good
    prm = backend.OptimizationAlgorithmFactory.instance().construct(solver)
    prm.initial_lambda = 1e-9
    prm.max_trials_after_failure = 4
    p = backend.CudaProblem(g, prm)
    before, chi0 = p.estimates(), p.chi2()
    for i in range(2):
        result, s = p.iterate(i)
        assert result == 2 and s["levenberg_iterations"] == 4
        assert all(np.array_equal(a, b) for a, b in zip(before, p.estimates()) if a is not None)
        assert p.chi2() == chi0 and s["chi2"] == pytest.approx(chi0[1], rel=1e-12)
    # and the context goes on from them
    g.information = good
    p.upload(g)
    q = backend.CudaProblem(g, prm)
    assert p.optimize(3)[0] == q.optimize(3)[0]
    assert all(np.array_equal(a, b) for a, b in zip(p.estimates(), q.estimates()) if a is not None)
