"""The stereo landmark pass and back-substitution by warps against the forms
with a thread per landmark, which a graph with a repeated observation takes."""

import copy

import numpy as np
import pytest

from g2o_b200 import synth

EPS = np.finfo(np.float64).eps


# one chunk of 32 edges, several, and landmarks of 2 to 20 edges
@pytest.mark.gpu
@pytest.mark.parametrize("cams,points,solver", [(3, 5, "lm_cuda"), (4, 60, "lm_cuda_chol"), (25, 700, "lm_cuda_chol"),
                                                (25, 700, "lm_cuda_mixed_fast")])
def test_both_forms(cams, points, solver):
    from g2o_b200 import backend
    g = synth.stereo_bundle_adjustment(cams, points, seed=cams)
    # a second observation of the first edge, without weight
    h = copy.deepcopy(g)
    h.edge_vertex = np.concatenate([g.edge_vertex, g.edge_vertex[:1]])
    h.measurement = np.concatenate([g.measurement, g.measurement[:1]])
    h.information = np.concatenate([g.information, np.zeros_like(g.information[:1])])
    if g.robust_delta is not None:
        h.robust_delta = np.concatenate([g.robust_delta, g.robust_delta[:1]])
    prm = backend.OptimizationAlgorithmFactory.instance().construct(solver)
    got = []
    for q in (g, h):
        p = backend.CudaProblem(q, prm)
        p.build_system()
        hpp, hll, hpl, b = p.hessian()
        status, x, _ = p.solve(1e4)
        assert status == 0
        got.append((hll, hpl, b, x))
    # float32 blocks are rounded once, the FP64 sums have at most 32 terms
    eps = 2.0 ** -23 if "mixed" in solver else EPS
    for a, c, e in zip(got[0][:3], got[1][:3], (eps, eps, EPS)):
        assert np.abs(a - c).max() <= 64 * e * np.abs(c).max()
    # the step: a damped system, its solves to 1e-6 of the residual norm at worst
    assert np.abs(got[0][3] - got[1][3]).max() <= 1e-4 * np.abs(got[1][3]).max()
