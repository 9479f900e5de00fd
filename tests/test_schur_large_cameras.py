"""Schur complements of graphs whose cameras' blocks do and do not fit in
shared memory, against the blocks they are made of."""

import numpy as np
import pytest

from g2o_b200 import synth

EPS = np.finfo(np.float64).eps


# about 1,350 FP64 blocks of one camera fit
@pytest.mark.gpu
@pytest.mark.parametrize("cams,points,odometry", [(3, 1200, False), (3, 1700, False), (5, 2500, False), (5, 2500, True),
                                                  (12, 3000, False), (20, 6000, True)])
def test_schur_matches_its_blocks(cams, points, odometry):
    from g2o_b200 import backend
    g = synth.bundle_adjustment(cams, points, seed=cams)
    if odometry:
        synth.add_odometry(g)
    p = backend.CudaProblem(g, backend.OptimizationAlgorithmFactory.instance().construct("lm_cuda"))
    p.build_system()
    lam = 50.0
    S, bs = p.schur(lam)
    hpp_rc, hpl_rc, rc = p.pattern()
    hpp, hll, hpl, b = p.hessian()
    nc, nl = p.info.num_free_poses, p.info.num_free_points
    W = np.zeros((nc * 6, nl * 3))
    for (r, c), v in zip(hpl_rc, hpl):
        c = c - nc if hpl_rc[:, 1].max() >= nl else c
        W[6 * r:6 * r + 6, 3 * c:3 * c + 3] = v
    D = np.linalg.inv(hll + lam * np.eye(3))
    WD = np.einsum("rlk,lkm->rlm", W.reshape(nc * 6, nl, 3), D).reshape(nc * 6, nl * 3)
    H = lam * np.eye(nc * 6)
    for (r, c), v in zip(hpp_rc, hpp):
        H[6 * r:6 * r + 6, 6 * c:6 * c + 6] += v
        if r != c:
            H[6 * c:6 * c + 6, 6 * r:6 * r + 6] += v.T
    want, rhs = H - WD @ W.T, b[:nc * 6] - WD @ b[nc * 6:]
    # sums of at most nl terms of this size, each of products of three
    tol = (nl + 64) * EPS * (np.abs(H).max() + (np.abs(WD) @ np.abs(W.T)).max())
    for (r, c), v in zip(rc, S):
        assert np.abs(v - want[6 * r:6 * r + 6, 6 * c:6 * c + 6]).max() <= tol
    assert np.abs(bs - rhs).max() <= (nl + 64) * EPS * (np.abs(b).max() + (np.abs(WD) @ np.abs(b[nc * 6:])).max())
    assert np.array_equal(S, p.schur(lam)[0])
