"""Marginals from the factor plan that the context keeps against those from a
plan made for the request, and contexts that follow one another or live on
several threads while sharing the cache of released device buffers."""

import threading

import numpy as np
import pytest

from g2o_b200 import synth

EPS = np.finfo(np.float64).eps


def construct(name):
    from g2o_b200 import backend
    return backend.OptimizationAlgorithmFactory.instance().construct(name)


# one tile, several separators; both block sizes; values held in float32 too
@pytest.mark.gpu
@pytest.mark.parametrize("kind,size,solver", [("2d", 4, "gn_cuda"), ("2d", 22, "gn_cuda"), ("2d", 300, "gn_cuda"),
                                              ("2d", 300, "gn_cuda_mixed"), ("3d", 4, "lm_cuda"), ("3d", 40, "lm_cuda_chol")])
def test_marginals_of_both_plans(kind, size, solver):
    from g2o_b200 import backend
    g = synth.pose_graph_2d(size, size // 3, seed=2) if kind == "2d" else synth.pose_graph_3d(3, size, seed=3)
    p = backend.CudaProblem(g, construct(solver))
    p.build_system()
    rc, H = p.pattern()[0], p.hessian()[0]
    nb, bs = p.info.num_free_poses, p.info.pose_dim
    dense = np.zeros((nb * bs, nb * bs))
    for (r, c), v in zip(rc, H):
        dense[r * bs:(r + 1) * bs, c * bs:(c + 1) * bs] = v
        dense[c * bs:(c + 1) * bs, r * bs:(r + 1) * bs] = v.T
    inv = np.linalg.inv(dense)
    # the bound of the inverse of a symmetric matrix by Cholesky, for both sides
    tol = 64 * nb * bs * EPS * np.linalg.cond(dense) * np.abs(inv).max()
    inside = np.concatenate([np.stack([np.arange(nb)] * 2, 1), rc, rc[:, ::-1]]).astype(np.int32)
    far = np.array([[0, nb - 1], [nb - 1, 0], [nb // 2, 0]], np.int32)
    a = p.compute_marginals(inside)
    b = p.compute_marginals(np.concatenate([inside, far]))
    for q, (r, c) in enumerate(np.concatenate([inside, far])):
        want = inv[r * bs:(r + 1) * bs, c * bs:(c + 1) * bs]
        assert np.abs(b[q] - want).max() <= tol
        if q < len(inside):
            assert np.abs(a[q] - want).max() <= tol
    assert np.array_equal(a, p.compute_marginals(inside))
    assert p.compute_marginals(np.zeros((0, 2), np.int32)).shape[0] == 0
    # the plan is still the solver's
    done, _ = p.optimize(2)
    q = backend.CudaProblem(g, construct(solver))
    assert q.optimize(2)[0] == done
    assert np.array_equal(p.estimates()[0], q.estimates()[0])


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [[[0, 99]], [[-1, 0]]])
def test_marginals_out_of_range(bad):
    from g2o_b200 import backend
    p = backend.CudaProblem(synth.pose_graph_2d(30, 8, seed=2), construct("gn_cuda"))
    with pytest.raises(Exception):
        p.compute_marginals(np.array(bad, np.int32))


@pytest.mark.gpu
def test_contexts_share_released_buffers():
    from g2o_b200 import backend
    graphs = [(synth.pose_graph_2d(150, 40, seed=1), "gn_cuda"), (synth.pose_graph_3d(3, 30, seed=2), "lm_cuda"),
              (synth.bundle_adjustment(8, 400, seed=3), "lm_cuda"),
              (synth.stereo_bundle_adjustment(8, 300, seed=4), "lm_cuda_chol")]

    def run(g, name):
        p = backend.CudaProblem(g, construct(name))
        p.optimize(3)
        e = p.estimates()
        p.close()
        return e

    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b) if x is not None)

    first = [run(*g) for g in graphs]
    assert all(same(run(*g), f) for _ in range(3) for g, f in zip(graphs, first))
    wrong = []

    def worker(k):
        for i in range(6):
            j = (k + i) % len(graphs)
            if not same(run(*graphs[j]), first[j]):
                wrong.append((k, j))

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
