"""Systems without full rank are refused and definite ones accepted, whatever
the size of their pivots: in the elimination order of a sparse graph the pivot
of a pose far from the fixed one is small in a definite system too."""

import numpy as np
import pytest

from g2o_b200 import synth

OK, NOT_PD = 0, 4


def problem(g, solver="gn_cuda"):
    from g2o_b200 import backend
    return backend.CudaProblem(g, backend.OptimizationAlgorithmFactory.instance().construct(solver))


def hinged(n, seed):
    """Two halves joined by one edge that does not see the heading: the second
    half may turn about its first pose."""
    g = synth.pose_graph_2d(n, n // 3, seed=seed)
    i, j = g.edge_vertex[:, 0], g.edge_vertex[:, 1]
    cut = n // 2
    keep = ~((i < cut) & (j >= cut) & (j != i + 1))
    for f in ("edge_vertex", "measurement", "information"):
        setattr(g, f, np.ascontiguousarray(getattr(g, f)[keep]))
    joint = np.flatnonzero((g.edge_vertex[:, 0] == cut - 1) & (g.edge_vertex[:, 1] == cut))
    info = g.information.reshape(-1, 3, 3)
    info[joint, 2, :] = 0.0
    info[joint, :, 2] = 0.0
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("n,seed", [(4, 0), (24, 1), (60, 0), (600, 2), (600, 3), (2000, 0), (2000, 1), (3500, 1),
                                    (3500, 2), (6000, 1), (10_000, 0), (20_000, 1)])
def test_free_heading_is_refused(n, seed):
    g = hinged(n, seed)
    p = problem(g)
    p.build_system()
    assert p.solve(0.0)[0] == NOT_PD
    assert p.solve(1.0)[0] == OK  # damped it is definite
    assert p.solve(0.0)[0] == NOT_PD
    if n <= 3500:
        from g2o_b200 import backend
        with pytest.raises(backend.G2ocError) as e:
            p.compute_marginals(np.array([[1, 1]], np.int32))
        assert e.value.status == NOT_PD


@pytest.mark.gpu
def test_free_gauge_is_refused_at_40000_poses():
    g = synth.pose_graph_2d(40_000, 13_333, seed=5)
    g.pose_fixed = np.zeros_like(g.pose_fixed)
    p = problem(g)
    p.build_system()
    assert p.solve(0.0)[0] == NOT_PD


# odometry alone: the farther from the fixed pose, the weaker the root's tie
@pytest.mark.gpu
@pytest.mark.parametrize("n,straight", [(3500, False), (20_000, False), (1000, True), (10_000, True)])
def test_weakly_tied_chain_is_accepted(n, straight):
    g = synth.pose_graph_2d(n, 0, seed=1)
    if straight:
        g.pose_estimate[:, 0] = np.arange(n)
        g.pose_estimate[:, 1:] = 0.0
        g.measurement = np.tile([1.0, 0.0, 0.0], (n - 1, 1))
    p = problem(g)
    p.build_system()
    assert p.solve(0.0)[0] == OK
    assert p.compute_marginals(np.array([[n // 2, n // 2]], np.int32))[0, 0, 0] > 0.0
