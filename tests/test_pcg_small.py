"""PCG solves of systems with few block rows: one cluster up to 64 rows (32 of
9 x 9), the grid-wide kernels beyond, against the dense system."""

import numpy as np
import pytest

from g2o_b200 import synth

TOL = 1e-12  # of r^T M^-1 r, relative to b^T M^-1 b


def preconditioned(A, bs, r):
    return sum(r[i:i + bs] @ np.linalg.solve(A[i:i + bs, i:i + bs], r[i:i + bs]) for i in range(0, len(r), bs))


def blocks(rc, vals, nb, bs):
    A = np.zeros((nb * bs, nb * bs))
    for (r, c), v in zip(rc, vals):
        A[r * bs:(r + 1) * bs, c * bs:(c + 1) * bs] = v
        A[c * bs:(c + 1) * bs, r * bs:(r + 1) * bs] = v.T
    return A


# the last column: block rows at the ends of a warp's lanes, a CTA's warps and the cluster
@pytest.mark.gpu
@pytest.mark.parametrize("kind,nb", [("2d", 1), ("2d", 8), ("2d", 33), ("2d", 64), ("2d", 65),
                                     ("3d", 11), ("3d", 32), ("3d", 62), ("3d", 65),
                                     ("ba", 1), ("ba", 7), ("ba", 8), ("ba", 9), ("ba", 32), ("ba", 33), ("ba", 64),
                                     ("ba", 65), ("mixed", 9), ("mixed", 33), ("bal", 3), ("bal", 32), ("bal", 33)])
def test_small_systems(kind, nb):
    from g2o_b200 import backend
    name = {"bal": "lm_cuda_pcg9_3", "mixed": "lm_cuda_mixed_fast"}.get(kind, "lm_cuda_pcg")
    prm = backend.OptimizationAlgorithmFactory.instance().construct(name)
    prm.pcg_tolerance = TOL
    prm.pcg_absolute_tolerance = 0
    lam = 1e3
    if kind == "2d":
        g = synth.pose_graph_2d(nb + 1, nb // 3, seed=nb)
    elif kind == "3d":
        g = synth.pose_graph_3d(3, (nb + 3) // 3, seed=nb)
    elif kind == "bal":
        g = synth.bal_problem(nb, 40 + 20 * nb, seed=nb)
    else:
        g = synth.bundle_adjustment(nb + 2, 40 + 20 * nb, seed=nb)
    p = backend.CudaProblem(g, prm)
    p.build_system()
    rows, bs = p.info.num_free_poses, p.info.pose_dim
    n = rows * bs
    if kind in ("2d", "3d"):
        A = blocks(p.pattern()[0], p.hessian()[0], rows, bs) + lam * np.eye(n)
        b = p.gradient()
    else:
        S, b = p.schur(lam)
        A = blocks(p.pattern()[2], S, rows, bs)
    status, x, its = p.solve(lam)
    assert status == 0 and 0 < its <= n
    r = b[:n] - A @ x[:n]
    # the residual that the iteration carries is within rounding of the true
    # one (float32 storage: of the rounded matrix, which is the one exported)
    assert preconditioned(A, bs, r) <= 4 * TOL * preconditioned(A, bs, b[:n])
    p.solver_init()
    again = p.solve(lam)
    assert again[2] == its and np.array_equal(again[1], x)
