"""An iteration that fails half-way (the all-reduce of a sharded run returns an
error): the call reports it, the iterations before it keep their statistics, and
the context goes on."""

import ctypes as C

import numpy as np
import pytest

from g2o_b200 import synth


class FailingReduce:
    """Rank 0's share is the whole graph, so the sum over the ranks is its own;
    the call after `left` more returns an error."""

    def __init__(self):
        self.calls, self.left = 0, None

    def __call__(self, ptr, count, dtype, op, stream):
        if self.left is not None:
            if self.left == 0:
                raise RuntimeError("all-reduce failed")
            self.left -= 1
        self.calls += 1


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["lm_cuda", "gn_cuda"])
@pytest.mark.parametrize("with_stats", [True, False])
def test_failure_after_good_iterations(solver, with_stats):
    from g2o_b200 import backend
    from g2o_b200.abi import G2ocIterationStats
    g = synth.bundle_adjustment(40, 1200, seed=3)
    reduce = FailingReduce()
    prm = backend.OptimizationAlgorithmFactory.instance().construct(solver)
    p = backend.CudaProblem(g, prm, shard=(0, 2, reduce))
    start = p.estimates()
    first = p.optimize(1)[1]
    per_iteration = reduce.calls
    assert per_iteration > 1
    L = backend.library()
    for more in range(1, per_iteration + 1):
        p.set_estimates(*start)
        reduce.left = per_iteration + more - 1
        stats = (G2ocIterationStats * 4)() if with_stats else None
        done = C.c_int()
        assert L.g2oc_optimize(p.handle, 4, stats, C.byref(done)) != 0
        if with_stats:
            assert stats[0].time_iteration > 0 and stats[0].time_quadratic_form > 0
            assert stats[0].chi2 == pytest.approx(first[0]["chi2"], rel=1e-9)
    reduce.left = None
    p.set_estimates(*start)
    good = backend.CudaProblem(g, prm, shard=(0, 2, FailingReduce()))
    assert p.optimize(3)[0] == good.optimize(3)[0] == 3
    assert all(np.array_equal(a, b) for a, b in zip(p.estimates(), good.estimates()))
