"""The end of an iteration: the chi2 that the last block of a grid-wide sum
forms and sends to the host, the errors carried over to the next iteration,
and the estimates restored from what the update kernel saved."""

import numpy as np
import pytest

from g2o_b200 import synth

EPS = np.finfo(np.float64).eps


def graph(kind, size):
    if kind == "2d":
        return synth.pose_graph_2d(size, size // 3, seed=5)
    if kind == "3d":
        return synth.pose_graph_3d(3, size, seed=6)
    if kind == "stereo":
        return synth.stereo_bundle_adjustment(6, size, seed=7)
    if kind == "bal":
        return synth.bal_problem(6, size, seed=8)
    return synth.bundle_adjustment(6, size, seed=9)


# edge counts on both sides of one block of 128 or 256 edges and, for the 2D
# graphs, beyond the grid that fills the GPU (592 x 256)
CASES = [("2d", 5, "gn_cuda"), ("2d", 190, "gn_cuda"), ("2d", 195, "lm_cuda"), ("2d", 120_000, "gn_cuda"),
         ("3d", 20, "gn_cuda"), ("3d", 60, "lm_cuda"), ("mono", 20, "lm_cuda"), ("mono", 900, "lm_cuda"),
         ("stereo", 300, "lm_cuda_chol"), ("bal", 200, "lm_cuda_pcg9_3")]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,size,solver", CASES)
def test_chi2_of_an_iteration_is_that_of_its_estimates(kind, size, solver):
    from g2o_b200 import backend
    g = graph(kind, size)
    prm = backend.OptimizationAlgorithmFactory.instance().construct(solver)
    its = 1 if size > 10_000 else 4
    p = backend.CudaProblem(g, prm)
    done, stats = p.optimize(its)
    assert len(stats) == done and all(s["time_iteration"] > 0 for s in stats)
    # sums of the same terms in some order
    tol = 4 * max(p.info.num_active_edges, 1) * EPS
    assert stats[-1]["chi2"] == pytest.approx(p.chi2()[1], rel=tol, abs=0)
    # one call or several: the same iterations, whether the errors are carried or computed
    q = backend.CudaProblem(g, prm)
    for i in range(done):
        _, s = q.iterate(i)
        assert s["chi2"] == stats[i]["chi2"]
        q.set_estimates(*q.estimates())
    assert all(np.array_equal(a, b) for a, b in zip(p.estimates(), q.estimates()) if a is not None)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,size,solver,sigma", [("2d", 190, "lm_cuda", 100.0), ("3d", 20, "lm_cuda", 100.0),
                                                    ("mono", 300, "lm_cuda", 100.0), ("mono", 300, "lm_cuda", 3.0),
                                                    ("stereo", 300, "lm_cuda_chol", 100.0),
                                                    ("bal", 200, "lm_cuda_pcg9_3", 1.0)])
def test_rejected_trials_leave_the_estimates(kind, size, solver, sigma):
    from g2o_b200 import backend
    g = graph(kind, size)
    rng = np.random.default_rng(3)
    est = {"2d": g.pose_estimate[1:], "3d": g.pose_estimate[1:, 9:], "bal": g.pose_estimate[:, :6]}.get(
        kind, g.point_estimate)
    est += rng.normal(0.0, sigma, est.shape)
    prm = backend.OptimizationAlgorithmFactory.instance().construct(solver)
    prm.initial_lambda = 1e-9
    p = backend.CudaProblem(g, prm)
    rejected = 0
    for i in range(8):
        before, chi0 = p.estimates(), p.chi2()[1]
        res, s = p.iterate(i)
        rejected += s["levenberg_iterations"] > 1
        after, chi1 = p.estimates(), p.chi2()[1]
        assert chi1 <= chi0
        assert s["chi2"] == pytest.approx(chi1, rel=4 * p.info.num_active_edges * EPS, abs=0)
        if chi1 == chi0:  # every trial was rejected
            assert all(np.array_equal(a, b) for a, b in zip(before, after) if a is not None)
        if res != 1:  # terminated
            break
    if rejected == 0:  # so far from the solution it can depend on rounding
        pytest.skip("no trial was rejected")
