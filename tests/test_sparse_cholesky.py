"""The tiled sparse Cholesky (nested-dissection plan, tiles computed by ticket)
through LinearSolver::solve and solvePattern on caller matrices: patterns and
sizes at the edges of its 64 x 64 tiles against dense FP64 linear algebra.

Tolerances: a Cholesky solve in FP64 with any summation order has a normwise
backward error of a few n eps (Higham, Accuracy and Stability of Numerical
Algorithms, theorem 10.4); with n <= 1200 and the sums cut into tiles, 64 n eps
leaves an order of magnitude. The matrices below are diagonally dominant, so
the inverse blocks (condition below 10) are held to the same figure relative
to the largest entry.
"""
import numpy as np
import pytest

EPS = 2.220446049250313e-16


def pattern(kind, nb, rng):
    pairs = set((i, i) for i in range(nb))

    def add(a, b):
        if a != b:
            pairs.add((min(a, b), max(a, b)))

    if kind == "chain":
        for i in range(nb - 1):
            add(i, i + 1)
    elif kind == "star":
        for i in range(1, nb):
            add(0, i)
    elif kind == "full":
        for i in range(nb):
            for j in range(i + 1, nb):
                add(i, j)
    elif kind == "grid":
        w = 9
        for i in range(nb):
            if i % w != w - 1 and i + 1 < nb:
                add(i, i + 1)
            if i + w < nb:
                add(i, i + w)
    elif kind == "islands":
        for i in range(nb - 1):
            if i % 7:
                add(i, i + 1)
    elif kind == "random":
        for a, b in rng.integers(0, nb, (2 * nb, 2)):
            add(int(a), int(b))
    return np.array(sorted(pairs, key=lambda p: (p[1], p[0])), np.int32)  # column-major


def system(kind, nb, bs, seed):
    rng = np.random.default_rng(seed)
    rc = pattern(kind, nb, rng)
    vals = rng.uniform(-1.0, 1.0, (len(rc), bs, bs))
    A = np.zeros((nb * bs, nb * bs))
    for k, (r, c) in enumerate(rc):
        if r == c:
            vals[k] = 0.5 * (vals[k] + vals[k].T)
        A[r * bs:(r + 1) * bs, c * bs:(c + 1) * bs] = vals[k]
        A[c * bs:(c + 1) * bs, r * bs:(r + 1) * bs] = vals[k].T
    # strictly dominant diagonal
    row = np.abs(A).sum(1)
    for k, (r, c) in enumerate(rc):
        if r == c:
            vals[k] += np.diag(1.5 * row[r * bs:(r + 1) * bs])
            A[r * bs:(r + 1) * bs, r * bs:(r + 1) * bs] = vals[k]
    return rc, vals, A, rng.uniform(-1.0, 1.0, nb * bs)


# n = nb * bs around one and two tiles of 64, and wide enough for several
# separators; the full pattern keeps the given order in one group (its largest
# here has more products per tile than are looked up at a time)
CASES = [("chain", 1, 3), ("chain", 21, 3), ("chain", 22, 3), ("chain", 10, 6), ("chain", 11, 6), ("chain", 400, 3),
         ("star", 43, 3), ("star", 150, 6), ("full", 11, 6), ("full", 43, 3), ("full", 60, 6), ("full", 190, 6),
         ("grid", 64, 3), ("grid", 199, 6), ("islands", 90, 3), ("islands", 33, 6), ("random", 130, 3), ("random", 77, 6)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nb,bs", CASES)
def test_solve_matches_dense(kind, nb, bs):
    from g2o_b200 import backend
    rc, vals, A, b = system(kind, nb, bs, seed=nb * 10 + bs)
    offs = np.arange(nb + 1, dtype=np.int32) * bs
    st, x, _ = backend.solve_block_system(backend.LINEAR_CHOLESKY, offs, rc, vals, b)
    assert st == 0
    n = nb * bs
    backward = np.linalg.norm(A @ x - b) / (np.linalg.norm(A, 2) * np.linalg.norm(x) + np.linalg.norm(b))
    assert backward <= 64 * n * EPS
    st2, x2, _ = backend.solve_block_system(backend.LINEAR_CHOLESKY, offs, rc, vals, b)
    assert st2 == 0 and np.array_equal(x, x2)  # the sums' order is the plan's


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nb,bs", [("chain", 1, 3), ("chain", 64, 3), ("star", 43, 6), ("full", 30, 6),
                                        ("grid", 150, 3), ("islands", 60, 3), ("random", 90, 6)])
def test_inverse_blocks_match_dense(kind, nb, bs):
    from g2o_b200 import backend
    rc, vals, A, _ = system(kind, nb, bs, seed=nb * 10 + bs + 1)
    rng = np.random.default_rng(nb)
    far = rng.integers(0, nb, (6, 2))  # pairs outside the pattern too
    req = np.concatenate([np.stack([np.arange(nb)] * 2, 1), far]).astype(np.int32)
    st, out = backend.solve_pattern_block_system(np.arange(nb + 1, dtype=np.int32) * bs, rc, vals, req)
    assert st == 0
    inv = np.linalg.inv(A)
    ref = np.stack([inv[r * bs:(r + 1) * bs, c * bs:(c + 1) * bs] for r, c in req])
    assert np.abs(out - ref).max() <= 64 * nb * bs * EPS * np.abs(inv).max()


@pytest.mark.gpu
def test_indefinite_matrix_is_reported():
    from g2o_b200 import abi, backend
    rc, vals, A, b = system("grid", 120, 3, seed=5)
    vals = vals.copy()
    vals[np.flatnonzero((rc[:, 0] == 77) & (rc[:, 1] == 77))[0]] *= -1.0
    st, _, _ = backend.solve_block_system(backend.LINEAR_CHOLESKY, np.arange(121, dtype=np.int32) * 3, rc, vals, b)
    assert abi.ERROR_NAMES[st] == "NOT_PD"


@pytest.mark.gpu
def test_wait_that_runs_out_is_an_error(monkeypatch):
    """A flag that nothing sets: the waits end, the call returns an error and
    the device stays usable."""
    from g2o_b200 import abi, backend, synth
    g = synth.pose_graph_2d(num_poses=60, num_closures=30, seed=2)
    prm = backend.OptimizationAlgorithmFactory.instance().construct("gn_cuda_chol")
    monkeypatch.setenv("G2OC_TEST_BARRIER_EXTRA", "1")
    c = backend.CudaProblem(g, prm)
    monkeypatch.delenv("G2OC_TEST_BARRIER_EXTRA")
    with pytest.raises(backend.G2ocError) as e:
        c.optimize(1)
    assert abi.ERROR_NAMES[e.value.status] == "TIMEOUT"
    good = backend.CudaProblem(g, prm)
    done, st = good.optimize(3)
    assert done == 3 and np.isfinite(st[-1]["chi2"])


# a chain's root is tied to the fixed pose by a pivot far below n eps of the
# largest entry; without the fixed pose the root's pivot is rounding alone
@pytest.mark.gpu
@pytest.mark.parametrize("poses,fixed,status", [(3400, True, 0), (40_000, True, 0), (60, False, 4), (3400, False, 4)])
def test_pivot_floor(poses, fixed, status):
    from g2o_b200 import backend, synth
    g = synth.pose_graph_2d(poses, poses // 3, seed=5)
    if not fixed:
        g.pose_fixed = np.zeros_like(g.pose_fixed)
    p = backend.CudaProblem(g, backend.OptimizationAlgorithmFactory.instance().construct("gn_cuda"))
    p.build_system()
    assert p.solve(0.0)[0] == status
