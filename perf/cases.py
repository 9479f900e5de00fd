"""The work a program that uses this library has it do, as cases to time.

Every case is one call sequence through the public Python entry points
(SparseOptimizer, CudaProblem, CudaWindows, BlockSolverCuda) on a graph of the
kinds and sizes the library's own configurations cover:

* pose graphs (VertexSE2 / EdgeSE2 Manhattan walks, VertexSE3 / EdgeSE3 rings)
  under Gauss-Newton and Levenberg-Marquardt with the sparse Cholesky, 60 to
  3,500 poses, and their marginal covariances;
* bundle adjustments (ring of cameras, box of points, Huber kernel, 1%
  outliers), 8 cameras and 200 points up to 1,000 cameras and 200,000 points,
  FP64 with the block-Jacobi PCG or the Cholesky, mono and stereo edges, and
  the mixed-precision form;
* a g2o host that drives the solve itself (buildSystem, setLambda, solve);
* batches of local windows;
* BAL problems (nine-parameter cameras).

The graphs come from seeded generators of the form of g2o_b200/synth.py; the
projection ones are drawn here with torch on the GPU, so that a graph of a
million edges is made in a fraction of a second. `exact` restates the same
iterations with dense linear algebra in torch float64.
"""
import math

import numpy as np
import torch

from g2o_b200 import abi, backend, synth

DEVICE = "cuda"
HUBER_MONO = math.sqrt(5.991)
HUBER_STEREO = math.sqrt(7.815)
FOCAL, WIDTH, HEIGHT = 500.0, 640, 480
STEREO_BF = 0.12 * FOCAL


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a robot's sliding 2D map: new measurements for the same graph, a few
        # Gauss-Newton steps, estimates back (latency of small solves)
        {"name": "pg2d_small", "kind": "pg2d", "poses": 203, "closures": 111, "solver": "gn_cuda", "iterations": 5,
         "reupload": True},
        # the Manhattan configuration: one full batch optimization
        {"name": "pg2d_manhattan", "kind": "pg2d", "poses": 3500, "closures": 2000, "solver": "gn_cuda",
         "iterations": 6, "reupload": False},
        # the sphere configuration under Levenberg-Marquardt
        {"name": "pg3d_sphere", "kind": "pg3d", "rings": 10, "per_ring": 250, "solver": "lm_cuda", "iterations": 4,
         "reupload": False},
        # a ragged medium 3D pose graph, as a back end re-optimizes it
        {"name": "pg3d_odd", "kind": "pg3d", "rings": 7, "per_ring": 61, "solver": "gn_cuda_chol", "iterations": 3,
         "reupload": True},
        # covariances of every pose of a 2D map (data association, gating)
        {"name": "pg2d_marginals", "kind": "marginals", "poses": 1201, "closures": 640},
        # local bundle adjustment at a keyframe: a new small graph through the
        # SparseOptimizer from construction to the estimates
        {"name": "ba_keyframe", "kind": "keyframe", "cameras": 11, "points": 417, "edge": "mono", "solver": "lm_cuda",
         "iterations": 5},
        # a medium local map solved exactly at each step (LinearSolverDense's role)
        {"name": "ba_cholesky", "kind": "ba", "cameras": 57, "points": 3001, "edge": "stereo",
         "solver": "lm_cuda_chol", "iterations": 4, "reupload": True},
        # one solve as a g2o host drives it: estimates in, b and x out
        {"name": "ba_adapter", "kind": "adapter", "cameras": 123, "points": 17003, "edge": "mono", "lam": 10.0},
        # the 1000-camera bundle adjustment, FP64
        {"name": "ba_large", "kind": "ba", "cameras": 1000, "points": 200000, "edge": "mono", "solver": "lm_cuda",
         "iterations": 6, "reupload": False},
        # the same in the mixed-precision form, the map held in float32 on the
        # GPU afterwards (dense mapping and rendering read it so)
        {"name": "ba_large_mixed", "kind": "ba", "cameras": 1000, "points": 200000, "edge": "mono",
         "solver": "lm_cuda_mixed_fast", "iterations": 6, "reupload": False},
        # many robots' local windows in one batch
        {"name": "windows_96", "kind": "windows", "windows": 96, "seed": 11, "solver": "lm_cuda", "iterations": 5},
        # a BAL problem of the Dubrovnik-356 shape at half its points
        {"name": "bal_356", "kind": "bal", "cameras": 356, "points": 113000, "solver": "lm_cuda_pcg9_3",
         "iterations": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pg2d", "pg2d", "pg3d", "pg3d", "marginals", "ba", "ba", "ba", "keyframe", "adapter", "windows",
                       "bal"])
    if kind == "pg2d":
        n = _log_uniform(rng, 60, 3400)
        return {"kind": kind, "poses": n, "closures": int(n * rng.uniform(0.3, 0.6)),
                "solver": rng.choice(["gn_cuda", "gn_cuda_chol", "lm_cuda"]), "iterations": rng.randint(2, 6),
                "reupload": rng.random() < 0.5}
    if kind == "pg3d":
        per = _log_uniform(rng, 20, 240)
        return {"kind": kind, "rings": rng.randint(3, 10), "per_ring": per,
                "solver": rng.choice(["gn_cuda", "lm_cuda", "lm_cuda_chol"]), "iterations": rng.randint(2, 4),
                "reupload": rng.random() < 0.5}
    if kind == "marginals":
        n = _log_uniform(rng, 60, 1200)
        return {"kind": kind, "poses": n, "closures": int(n * rng.uniform(0.3, 0.6))}
    if kind == "keyframe":
        return {"kind": kind, "cameras": rng.randint(8, 30), "points": _log_uniform(rng, 200, 3000),
                "edge": rng.choice(["mono", "stereo"]), "solver": rng.choice(["lm_cuda", "lm_cuda_chol"]),
                "iterations": rng.randint(3, 6)}
    if kind == "adapter":
        cams = _log_uniform(rng, 20, 400)
        return {"kind": kind, "cameras": cams, "points": _log_uniform(rng, 30 * cams, 150 * cams),
                "edge": rng.choice(["mono", "stereo"]), "lam": float(rng.choice([1.0, 10.0, 100.0]))}
    if kind == "windows":
        return {"kind": kind, "windows": _log_uniform(rng, 4, 90), "seed": rng.randrange(1 << 20),
                "solver": "lm_cuda", "iterations": rng.randint(3, 5)}
    if kind == "bal":
        cams = _log_uniform(rng, 20, 340)
        return {"kind": kind, "cameras": cams, "points": _log_uniform(rng, 60 * cams, 300 * cams),
                "solver": "lm_cuda_pcg9_3", "iterations": rng.randint(2, 3)}
    solver = rng.choice(["lm_cuda", "lm_cuda", "lm_cuda_chol", "lm_cuda_mixed_fast"])
    cams = _log_uniform(rng, 12, 110 if solver == "lm_cuda_chol" else 950)
    return {"kind": kind, "cameras": cams, "points": _log_uniform(rng, 40 * cams, 190 * cams),
            "edge": rng.choice(["mono", "stereo"]), "solver": solver, "iterations": rng.randint(3, 6),
            "reupload": rng.random() < 0.5}


# -------------------------------------------------------------- generators
def _scene(cameras, points, seed, max_obs=20, mean_obs=5.0, min_obs=2):
    """Ring of inward-looking cameras around a box of points and who sees
    what: every point gets a truncated geometric number of observations among
    the cameras that have it in the image. Edges by point, then by camera.
    (float64 torch tensors on the GPU; synth.bundle_adjustment's scene)"""
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed) * 1000003 + 17)
    f64 = dict(device=DEVICE, dtype=torch.float64)
    az = 2 * math.pi * torch.arange(cameras, **f64) / cameras
    centre = torch.stack([30.0 * torch.cos(az), 30.0 * torch.sin(az), torch.full_like(az, 1.5)], 1)
    fwd = torch.tensor([0.0, 0.0, 2.5], **f64) - centre
    fwd = fwd / fwd.norm(dim=1, keepdim=True)
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 0.0, 1.0], **f64).expand_as(fwd))
    right = right / right.norm(dim=1, keepdim=True)
    R = torch.stack([right, torch.linalg.cross(fwd, right), fwd], 1)
    t = -(R @ centre[:, :, None])[:, :, 0]
    lo = torch.tensor([-10.0, -10.0, 0.0], **f64)
    size = torch.tensor([20.0, 20.0, 5.0], **f64)
    X = lo + size * torch.rand((points, 3), generator=gen, **f64)
    m = min(max_obs, cameras)
    u = torch.rand(points, generator=gen, **f64)
    k = 1 + torch.floor(torch.log1p(-u) / math.log(1.0 - 1.0 / mean_obs)).clamp(0, 1000).long()
    k = k.clamp(min(min_obs, m), m)
    pts, cams, uvs, depth = [], [], [], []
    step = max(1, (1 << 25) // cameras)
    for s in range(0, points, step):
        Xs = X[s:s + step]
        Xc = torch.einsum("cij,pj->pci", R, Xs) + t
        uv = FOCAL * Xc[..., :2] / Xc[..., 2:] + torch.tensor([WIDTH / 2.0, HEIGHT / 2.0], **f64)
        vis = (Xc[..., 2] > 0.5) & (uv[..., 0] >= 0) & (uv[..., 0] < WIDTH) & (uv[..., 1] >= 0) & (uv[..., 1] < HEIGHT)
        key = torch.rand(vis.shape, generator=gen, device=DEVICE).masked_fill_(~vis, 2.0)
        best, cand = torch.topk(key, m, dim=1, largest=False)
        ks = torch.minimum(k[s:s + step], vis.sum(1))
        ks = torch.where(ks < 2, torch.zeros_like(ks), ks)
        cand = torch.where(torch.arange(m, device=DEVICE)[None, :] < ks[:, None], cand, cameras).sort(dim=1).values
        row, col = torch.nonzero(cand < cameras, as_tuple=True)
        c = cand[row, col]
        pts.append(s + row)
        cams.append(c)
        uvs.append(uv[row, c])
        depth.append(Xc[row, c, 2])
    pts, cams, uv, z = torch.cat(pts), torch.cat(cams), torch.cat(uvs), torch.cat(depth)
    used, pts = torch.unique(pts, return_inverse=True)
    return gen, R, t, X[used], pts, cams, uv, z


def _quat(R):
    return torch.from_numpy(synth._rot_to_quat(R.cpu().numpy())).to(DEVICE)


def _rodrigues(v):
    th = v.norm(dim=1)[:, None, None].clamp_min(1e-300)
    K = _skew(v)
    return torch.eye(3, device=v.device, dtype=v.dtype) + torch.sin(th) / th * K + (1 - torch.cos(th)) / (th * th) * (K @ K)


def _ba_graph(cameras, points, edge, seed, max_obs=20, mean_obs=5.0):
    gen, R, t, X, pts, cams, uv, z = _scene(cameras, points, seed, max_obs, mean_obs)
    E = len(pts)

    def normal(shape, sigma):
        return sigma * torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float64)

    clean = uv[:, 0]
    uv = uv + normal((E, 2), 1.0)
    out = torch.rand(E, generator=gen, device=DEVICE) < 0.01
    anywhere = torch.rand((E, 2), generator=gen, device=DEVICE, dtype=torch.float64)
    uv = torch.where(out[:, None], anywhere * torch.tensor([WIDTH, HEIGHT], device=DEVICE, dtype=torch.float64), uv)
    dR, dt = _rodrigues(normal((cameras, 3), 0.01)), normal((cameras, 3), 0.05)
    fixed = np.zeros(cameras, np.uint8)
    fixed[:2] = 1
    dR[:2] = torch.eye(3, device=DEVICE, dtype=torch.float64)
    dt[:2] = 0.0
    pose = torch.cat([(dR @ t[:, :, None])[:, :, 0] + dt, _quat(dR @ R)], 1)
    X0 = X + normal(X.shape, 0.1)
    meas, D, delta = uv, 2, HUBER_MONO
    if edge == "stereo":
        meas, D, delta = torch.cat([uv, (clean - STEREO_BF / z + normal((E,), 0.5))[:, None]], 1), 3, HUBER_STEREO
    return abi.Graph(abi.POSE_SE3EXPMAP,
                     abi.EDGE_STEREO_SE3_PROJECT_XYZ if edge == "stereo" else abi.EDGE_PROJECT_XYZ2UV,
                     pose.cpu().numpy(), torch.stack([pts, cams], 1).int().cpu().numpy(), meas.cpu().numpy(),
                     np.tile(np.eye(D).reshape(1, D * D), (E, 1)), pose_fixed=fixed, point_estimate=X0.cpu().numpy(),
                     point_fixed=np.zeros(len(X), np.uint8), robust_delta=np.full(E, delta), focal_length=FOCAL,
                     principal_point=(WIDTH / 2.0, HEIGHT / 2.0), focal_length_y=FOCAL if edge == "stereo" else None,
                     stereo_bf=STEREO_BF if edge == "stereo" else 0.0)


def _bal_graph(cameras, points, seed):
    gen, R, t, X, pts, cams, _, _ = _scene(cameras, points, seed, mean_obs=5.5)
    rng = np.random.default_rng(seed + 104729)
    flip = torch.tensor([1.0, -1.0, -1.0], device=DEVICE, dtype=torch.float64)
    cam = np.empty((cameras, 9))
    cam[:, 0:3] = synth._rot_to_angle_axis((flip[:, None] * R).cpu().numpy())
    cam[:, 3:6] = (flip * t).cpu().numpy()
    cam[:, 6] = FOCAL * (1.0 + rng.uniform(-0.02, 0.02, cameras))
    cam[:, 7] = rng.uniform(-0.05, 0.05, cameras)
    cam[:, 8] = rng.uniform(-0.01, 0.01, cameras)
    E = len(pts)
    ct = torch.from_numpy(cam).to(DEVICE)
    meas = _bal_project(ct[cams], X[pts]) + torch.randn((E, 2), generator=gen, device=DEVICE, dtype=torch.float64)
    X0 = X + 0.1 * torch.randn(X.shape, generator=gen, device=DEVICE, dtype=torch.float64)
    cam[:, 0:3] += rng.normal(0.0, 0.01, size=(cameras, 3))
    cam[:, 3:6] += rng.normal(0.0, 0.05, size=(cameras, 3))
    cam[:, 6] *= 1.0 + rng.normal(0.0, 0.01, cameras)
    cam[:, 7:9] = 0.0
    return abi.Graph(abi.POSE_BAL_CAMERA, abi.EDGE_BAL_OBSERVATION, cam,
                     torch.stack([pts, cams], 1).int().cpu().numpy(), meas.cpu().numpy(),
                     np.tile(np.eye(2).reshape(1, 4), (E, 1)), pose_fixed=np.zeros(cameras, np.uint8),
                     point_estimate=X0.cpu().numpy(), point_fixed=np.zeros(len(X), np.uint8))


def _window_sizes(case):
    return synth.window_sizes(case["windows"], seed=case["seed"])


def _graph(case, seed):
    kind = case["kind"]
    if kind in ("pg2d", "marginals"):
        return synth.pose_graph_2d(case["poses"], case["closures"], seed=seed)
    if kind == "pg3d":
        return synth.pose_graph_3d(case["rings"], case["per_ring"], seed=seed)
    if kind == "bal":
        return _bal_graph(case["cameras"], case["points"], seed)
    return _ba_graph(case["cameras"], case["points"], case["edge"], seed)


def _window_graphs(case, seed):
    return [_ba_graph(c, p, "mono", seed * 4099 + w, max_obs=8) for w, (c, p) in enumerate(_window_sizes(case))]


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    kind = case["kind"]
    params = None
    if "solver" in case:
        params = backend.OptimizationAlgorithmFactory.instance().construct(case["solver"])
    if kind == "windows":
        return {"case": case, "windows": backend.CudaWindows(_window_graphs(case, seed), params)}
    graph = _graph(case, seed)
    if kind == "keyframe":
        # the optimizer updates its graph's estimates in place
        return {"case": case, "graph": graph, "params": params, "pose": graph.pose_estimate.copy(),
                "point": graph.point_estimate.copy()}
    if kind == "adapter":
        solver = backend.BlockSolverCuda(backend.LinearSolverCudaPCG())
        solver.init(graph)
        solver.build_structure()
        return {"case": case, "graph": graph, "solver": solver}
    problem = backend.CudaProblem(graph, params)
    if kind == "marginals":
        free = np.arange(case["poses"] - 1, dtype=np.int32)
        return {"case": case, "problem": problem, "blocks": np.stack([free, free], 1)}
    return {"case": case, "graph": graph, "problem": problem}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "windows":
        w = state["windows"]
        w.restore_initial_estimates()
        stats = w.optimize(case["iterations"])
        est = w.estimates_all()
        return {"pose": np.concatenate([p for p, _ in est]), "point": np.concatenate([q for _, q in est]),
                "iterations": np.array([s["iterations"] for s in stats], np.int64)}
    if kind == "keyframe":
        g = state["graph"]
        g.pose_estimate[...] = state["pose"]
        g.point_estimate[...] = state["point"]
        opt = backend.SparseOptimizer()
        opt.set_algorithm(state["params"])
        opt.set_graph(g)
        opt.initialize_optimization()
        done = opt.optimize(case["iterations"])
        return {"pose": g.pose_estimate, "point": g.point_estimate, "iterations": done}
    if kind == "adapter":
        g, solver = state["graph"], state["solver"]
        solver.init(g)
        solver.build_system(g.pose_estimate, g.point_estimate)
        solver.set_lambda(case["lam"])
        solver.solve()
        solver.restore_diagonal()
        return {"b": solver.b(), "x": solver.x()}
    problem = state["problem"]
    if kind == "marginals":
        return problem.compute_marginals(state["blocks"])
    if case.get("reupload"):
        problem.upload(state["graph"])
    else:
        problem.restore_initial_estimates()
    done, _ = problem.optimize(case["iterations"])
    pose, point = problem.estimates()
    if kind == "ba" and "mixed" in case["solver"]:
        return {"pose": torch.from_numpy(pose).to(DEVICE, torch.float32),
                "point": torch.from_numpy(point).to(DEVICE, torch.float32), "iterations": done}
    return {"pose": pose, "point": point, "iterations": done}


# -------------------------------------------------------------------- work
def _mean_obs(cameras, max_obs=20, mean=5.0):
    """Mean of the geometric number of observations cut to [2, max]."""
    m = min(max_obs, cameras)
    q = 1.0 - 1.0 / mean
    return 1.0 + sum(q ** k for k in range(1, m)) + 1.0 / mean


def _ba_work(cameras, points, D, dim, iterations, per_point, pcg_iterations=12.0, real=8.0):
    """Per iteration: every edge's measurement and both its ends read for the
    linearization and for the chi2 of the trial, the Hessian blocks written
    and read once by the Schur complement and once by the back-substitution,
    the reduced camera system written and read once, the estimates updated."""
    E, P, C = points * per_point, points, cameras
    pairs = P * 0.5 * per_point * per_point
    blocks = min(0.5 * C * C, pairs) + C
    nbytes = 2 * E * (8 * D + 8) + E * 3 * dim * real * 3 + P * (6 + 9 + 24) * real + blocks * dim * dim * real * 2
    flops = E * (200 + 2 * D * (dim * dim + 3 * dim + 9)) + pairs * 2 * 3 * dim * dim + E * 2 * 9 * dim
    flops += pcg_iterations * 2 * 2 * blocks * dim * dim
    return iterations * nbytes, iterations * flops


def work(case):
    kind = case["kind"]
    if kind in ("pg2d", "pg3d", "marginals"):
        n, d, md = (case["rings"] * case["per_ring"], 6, 12) if kind == "pg3d" else (case["poses"], 3, 3)
        edges = 2.0 * n if kind == "pg3d" else n + case["closures"]
        # factor of a planar graph in nested-dissection order: about
        # 7.75 n log2 n block entries, (829 / 84) n^1.5 block products
        # (George 1973), each block d x d; the factor is written and read once
        # per direction of the substitution
        fill = 7.75 * n * math.log2(max(n, 4)) * 0.25
        factor = 9.87 * n ** 1.5 * 0.25
        its = case.get("iterations", 1)
        nbytes = its * (edges * 8 * (md + d * d + 4) * 2 + (n + edges) * d * d * 8 * 2 + fill * d * d * 8 * 3
                        + n * md * 8 * 3)
        flops = its * (edges * 12 * d ** 3 + factor * 2 * d ** 3 + 4 * fill * d * d)
        if kind == "marginals":
            nbytes += n * d * d * 8 + fill * d * d * 8
            flops += 2 * factor * 2 * d ** 3
        return {"bytes": nbytes, "flops": flops}
    if kind == "windows":
        total = [0.0, 0.0]
        for c, p in _window_sizes(case):
            b, f = _ba_work(c, p, 2, 6, case["iterations"], _mean_obs(c, 8), 0.0)
            total[0] += b
            total[1] += f + case["iterations"] * (6.0 * c) ** 3 / 3
        return {"bytes": total[0], "flops": total[1]}
    if kind == "bal":
        b, f = _ba_work(case["cameras"], case["points"], 2, 9, case["iterations"], _mean_obs(case["cameras"], 20, 5.5))
        return {"bytes": b, "flops": f}
    D = 3 if case["edge"] == "stereo" else 2
    real = 4.0 if "mixed" in case.get("solver", "") else 8.0
    b, f = _ba_work(case["cameras"], case["points"], D, 6, case.get("iterations", 1), _mean_obs(case["cameras"]),
                    real=real)
    if "chol" in case.get("solver", ""):
        f += case["iterations"] * (6.0 * case["cameras"]) ** 3 / 3
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact
def _skew(v):
    z = torch.zeros_like(v[..., 0])
    return torch.stack([torch.stack([z, -v[..., 2], v[..., 1]], -1), torch.stack([v[..., 2], z, -v[..., 0]], -1),
                        torch.stack([-v[..., 1], v[..., 0], z], -1)], -2)


def _rot(q):
    x, y, z, w = q.unbind(-1)
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
        torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], -2)


def _qmul(a, b):
    v = a[..., 3:] * b[..., :3] + b[..., 3:] * a[..., :3] + torch.linalg.cross(a[..., :3], b[..., :3])
    return torch.cat([v, (a[..., 3] * b[..., 3] - (a[..., :3] * b[..., :3]).sum(-1))[..., None]], -1)


def _bal_project(cam, X):
    w, t, f, k1, k2 = cam[..., 0:3], cam[..., 3:6], cam[..., 6], cam[..., 7], cam[..., 8]
    th = torch.sqrt((w * w).sum(-1, keepdim=True))
    v = w / th
    P = X * torch.cos(th) + torch.linalg.cross(v, X) * torch.sin(th) + v * (v * X).sum(-1, keepdim=True) * (1 - torch.cos(th)) + t
    p = -P[..., :2] / P[..., 2:]
    r2 = (p * p).sum(-1)
    return (f * (1 + k1 * r2 + k2 * r2 * r2))[..., None] * p


def _bal_model(cam, X, z):
    """Errors and Jacobians of EdgeObservationBAL."""
    err = lambda c, x, m: _bal_project(c, x) - m  # noqa: E731
    Jc, Jp = torch.func.vmap(torch.func.jacfwd(err, argnums=(0, 1)))(cam, X, z)
    return err(cam, X, z), Jp, Jc


def _ba_model(cam, X, z):
    """Errors and Jacobians of the mono and stereo projections; camera update
    T <- exp(omega, upsilon) T."""
    R = _rot(cam[:, 3:])
    P = (R @ X[:, :, None])[:, :, 0] + cam[:, :3]
    x, y, d = P.unbind(-1)
    o = torch.zeros_like(x)
    rows = [torch.stack([FOCAL / d, o, -FOCAL * x / (d * d)], -1), torch.stack([o, FOCAL / d, -FOCAL * y / (d * d)], -1)]
    pred = [FOCAL * x / d + WIDTH / 2.0, FOCAL * y / d + HEIGHT / 2.0]
    if z.shape[1] == 3:
        rows.append(torch.stack([FOCAL / d, o, -FOCAL * x / (d * d) + STEREO_BF / (d * d)], -1))
        pred.append(pred[0] - STEREO_BF / d)
    J = torch.stack(rows, 1)
    return z - torch.stack(pred, 1), -J @ R, torch.cat([J @ _skew(P), -J], 2)


def _ba_oplus(cam, dx):
    """SE3Quat::exp([omega, upsilon]) times the camera."""
    w, u = dx[:, :3], dx[:, 3:]
    th = w.norm(dim=1)
    safe = th.clamp_min(1e-300)
    K = _skew(w)
    A = ((1 - torch.cos(safe)) / (safe * safe))[:, None, None]
    B = ((safe - torch.sin(safe)) / safe ** 3)[:, None, None]
    small = (th < 1e-5)[:, None, None]
    V = torch.eye(3, device=cam.device, dtype=cam.dtype) + torch.where(small, 0.5 * K + K @ K / 6, A * K + B * (K @ K))
    q = torch.cat([w * (torch.sin(safe / 2) / safe)[:, None], torch.cos(th / 2)[:, None]], 1)
    t = (_rot(q) @ cam[:, :3, None])[:, :, 0] + (V @ u[:, :, None])[:, :, 0]
    q = _qmul(q, cam[:, 3:])
    q = q / q.norm(dim=1, keepdim=True)
    return torch.cat([t, torch.where(q[:, 3:] < 0, -q, q)], 1)


class _BA:
    """Normal equations of a projection graph: Huber-weighted, landmarks
    eliminated, reduced camera system dense."""

    def __init__(self, g):
        on = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)  # noqa: E731
        self.bal = g.edge_type == abi.EDGE_BAL_OBSERVATION
        self.dim = 9 if self.bal else 6
        self.pts, self.cams = on(g.edge_vertex[:, 0]).long(), on(g.edge_vertex[:, 1]).long()
        self.z = on(g.measurement)
        self.delta = None if g.robust_delta is None else on(g.robust_delta)
        self.x = (on(g.pose_estimate), on(g.point_estimate))
        self.C, self.P = g.num_poses, g.num_points
        self.free = on(g.pose_fixed) == 0

    def model(self, x):
        return (_bal_model if self.bal else _ba_model)(x[0][self.cams], x[1][self.pts], self.z)

    def chi2(self, x):
        if self.bal:
            e = _bal_project(x[0][self.cams], x[1][self.pts]) - self.z
        else:
            e = _ba_model(x[0][self.cams], x[1][self.pts], self.z)[0]
        s = (e * e).sum(1)
        if self.delta is None:
            return float(s.sum())
        return float(torch.where(s <= self.delta ** 2, s, 2 * s.sqrt() * self.delta - self.delta ** 2).sum())

    def linearize(self):
        e, Jp, Jc = self.model(self.x)
        s = (e * e).sum(1)
        w = torch.ones_like(s) if self.delta is None else torch.where(s <= self.delta ** 2, torch.ones_like(s), self.delta / s.sqrt())
        d, C, P = self.dim, self.C, self.P
        Jp_w, Jc_w = Jp * w[:, None, None], Jc * w[:, None, None]
        zeros = lambda *n: torch.zeros(n, device=DEVICE, dtype=torch.float64)  # noqa: E731
        self.Hpp = zeros(C, d, d).index_add_(0, self.cams, Jc_w.transpose(1, 2) @ Jc)
        self.Hll = zeros(P, 3, 3).index_add_(0, self.pts, Jp_w.transpose(1, 2) @ Jp)
        self.W = (Jc_w.transpose(1, 2) @ Jp) * self.free[self.cams][:, None, None]
        self.bp = -zeros(C, d).index_add_(0, self.cams, (Jc_w.transpose(1, 2) @ e[:, :, None])[:, :, 0]) * self.free[:, None]
        self.bl = -zeros(P, 3).index_add_(0, self.pts, (Jp_w.transpose(1, 2) @ e[:, :, None])[:, :, 0])

    def max_diag(self):
        a = self.Hpp[self.free].diagonal(dim1=1, dim2=2).abs().max()
        return float(torch.maximum(a, self.Hll.diagonal(dim1=1, dim2=2).abs().max()))

    def solve(self, lam):
        d, C = self.dim, self.C
        eye = lambda n: torch.eye(n, device=DEVICE, dtype=torch.float64)  # noqa: E731
        Dinv = torch.linalg.inv(self.Hll + lam * eye(3))
        Y = self.W @ Dinv[self.pts]
        S = torch.zeros((C * C, d, d), device=DEVICE, dtype=torch.float64)
        ar = torch.arange(C, device=DEVICE)
        S.index_add_(0, ar * C + ar, self.Hpp + lam * eye(d))
        E = len(self.pts)
        for k in range(E):  # edges are sorted by point: the k-th next edge of the same point
            a = torch.nonzero(self.pts[: E - k] == self.pts[k:]).squeeze(1)
            if len(a) == 0:
                break
            blk = -(Y[a] @ self.W[a + k].transpose(1, 2))
            S.index_add_(0, self.cams[a] * C + self.cams[a + k], blk)
            if k:
                S.index_add_(0, self.cams[a + k] * C + self.cams[a], blk.transpose(1, 2))
        S = S.view(C, C, d, d).permute(0, 2, 1, 3)
        S = S[self.free][:, :, self.free]
        n = S.shape[0] * d
        r = self.bp.index_add(0, self.cams, -(Y @ self.bl[self.pts][:, :, None])[:, :, 0])[self.free].reshape(-1, 1)
        xp = torch.zeros_like(self.bp)
        xp[self.free] = torch.cholesky_solve(r, torch.linalg.cholesky(S.reshape(n, n))).view(-1, d)
        back = self.bl.index_add(0, self.pts, -(self.W.transpose(1, 2) @ xp[self.cams][:, :, None])[:, :, 0])
        return xp, (Dinv @ back[:, :, None])[:, :, 0]

    def gain_scale(self, dx, lam):
        return float((dx[0] * (lam * dx[0] + self.bp)).sum() + (dx[1] * (lam * dx[1] + self.bl)).sum())

    def moved(self, dx):
        cam = self.x[0] + dx[0] if self.bal else torch.where(self.free[:, None], _ba_oplus(self.x[0], dx[0]), self.x[0])
        return cam, self.x[1] + dx[1]


def _se2_error(xi, xj, z):
    c, s = torch.cos(xi[2]), torch.sin(xi[2])
    dx, dy = xj[0] - xi[0], xj[1] - xi[1]
    rx, ry = c * dx + s * dy - z[0], -s * dx + c * dy - z[1]
    cz, sz = torch.cos(z[2]), torch.sin(z[2])
    a = xj[2] - xi[2] - z[2]
    return torch.stack([cz * rx + sz * ry, -sz * rx + cz * ry, torch.atan2(torch.sin(a), torch.cos(a))])


def _se2_plus(x, d):
    return x + d


def _compact(R):
    """Vector part of a rotation's quaternion with w >= 0."""
    w = 0.5 * torch.sqrt(1.0 + R[0, 0] + R[1, 1] + R[2, 2])
    return torch.stack([R[2, 1] - R[1, 2], R[0, 2] - R[2, 0], R[1, 0] - R[0, 1]]) / (4 * w)


def _se3_error(xi, xj, z):
    Ri, Rj, Rz = xi[:9].view(3, 3), xj[:9].view(3, 3), z[:9].view(3, 3)
    t = Rz.T @ (Ri.T @ (xj[9:] - xi[9:]) - z[9:])
    return torch.cat([t, _compact(Rz.T @ (Ri.T @ Rj))])


def _se3_plus(x, d):
    R = x[:9].view(3, 3)
    q = torch.cat([d[3:], torch.sqrt(1.0 - (d[3:] * d[3:]).sum())[None]])
    return torch.cat([(R @ _rot(q)).reshape(-1), x[9:] + R @ d[:3]])


class _PG:
    """Normal equations of a pose graph, dense."""

    def __init__(self, g):
        on = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)  # noqa: E731
        self.dim = 3 if g.pose_type == abi.POSE_SE2 else 6
        self.error, self.plus = (_se2_error, _se2_plus) if self.dim == 3 else (_se3_error, _se3_plus)
        self.i, self.j = on(g.edge_vertex[:, 0]).long(), on(g.edge_vertex[:, 1]).long()
        self.z = on(g.measurement)
        self.omega = on(g.information).view(len(self.z), self.dim, self.dim)
        self.x = on(g.pose_estimate)
        self.free = on(g.pose_fixed) == 0
        self.n = len(self.x)

    def chi2(self, x):
        e = torch.func.vmap(self.error)(x[self.i], x[self.j], self.z)
        return float((e * (self.omega @ e[:, :, None])[:, :, 0]).sum())

    def linearize(self):
        d, n = self.dim, self.n
        f = lambda a, b, xi, xj, z: self.error(self.plus(xi, a), self.plus(xj, b), z)  # noqa: E731
        o = torch.zeros((len(self.z), d), device=DEVICE, dtype=torch.float64)
        args = (o, o, self.x[self.i], self.x[self.j], self.z)
        e = torch.func.vmap(self.error)(*args[2:])
        Ji, Jj = torch.func.vmap(torch.func.jacfwd(f, argnums=(0, 1)))(*args)
        H = torch.zeros((n * n, d, d), device=DEVICE, dtype=torch.float64)
        b = torch.zeros((n, d), device=DEVICE, dtype=torch.float64)
        for u, Ju in ((self.i, Ji), (self.j, Jj)):
            JO = Ju.transpose(1, 2) @ self.omega
            b.index_add_(0, u, -(JO @ e[:, :, None])[:, :, 0])
            for v, Jv in ((self.i, Ji), (self.j, Jj)):
                H.index_add_(0, u * n + v, JO @ Jv)
        H = H.view(n, n, d, d).permute(0, 2, 1, 3)[self.free][:, :, self.free]
        self.H = H.reshape(H.shape[0] * d, -1)
        self.b = b[self.free].reshape(-1, 1)

    def max_diag(self):
        return float(self.H.diagonal().abs().max())

    def factor(self, lam):
        H = self.H.clone()
        H.diagonal().add_(lam)
        return torch.linalg.cholesky(H)

    def solve(self, lam):
        return torch.cholesky_solve(self.b, self.factor(lam))

    def gain_scale(self, dx, lam):
        return float((dx * (lam * dx + self.b)).sum())

    def moved(self, dx):
        d = torch.zeros((self.n, self.dim), device=DEVICE, dtype=torch.float64)
        d[self.free] = dx.view(-1, self.dim)
        x = torch.func.vmap(self.plus)(self.x, d)
        if self.dim == 3:
            x = torch.cat([x[:, :2], torch.atan2(torch.sin(x[:, 2:]), torch.cos(x[:, 2:]))], 1)
        return torch.where(self.free[:, None], x, self.x)


def _gauss_newton(sys, iterations):
    for _ in range(iterations):
        sys.linearize()
        sys.x = sys.moved(sys.solve(0.0))


def _levenberg(sys, iterations):
    """OptimizationAlgorithmLevenberg::solve; the iterations completed."""
    lam, ni, done = 0.0, 2.0, 0
    for it in range(iterations):
        sys.linearize()
        current = sys.chi2(sys.x)
        if it == 0:
            lam, ni = 1e-5 * sys.max_diag(), 2.0
        rho, tries = -1.0, 0
        while rho < 0 and tries < 10:
            dx = sys.solve(lam)
            x = sys.moved(dx)
            chi2 = sys.chi2(x)
            rho = (current - chi2) / (sys.gain_scale(dx, lam) + 1e-3)
            if rho > 0 and math.isfinite(chi2):
                lam, ni, sys.x = lam * max(1 / 3, min(2 / 3, 1 - (2 * rho - 1) ** 3)), 2.0, x
            else:
                lam, ni = lam * ni, ni * 2
            tries += 1
        done += 1
        if tries == 10 or rho == 0 or not math.isfinite(lam):
            break
    return done


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pg2d", "pg3d", "marginals"):
        s = _PG(_graph(case, seed))
        if kind == "marginals":
            s.linearize()
            inv = torch.cholesky_inverse(s.factor(0.0))
            m = inv.shape[0] // 3
            return inv.view(m, 3, m, 3).permute(0, 2, 1, 3)[torch.arange(m), torch.arange(m)].cpu().numpy()
        if case["solver"].startswith("gn"):
            _gauss_newton(s, case["iterations"])
        else:
            _levenberg(s, case["iterations"])
        return {"pose": s.x.cpu().numpy(), "point": None, "iterations": None}
    if kind == "windows":
        done = []
        for g in _window_graphs(case, seed):
            s = _BA(g)
            _levenberg(s, case["iterations"])
            done.append(s.x)
        return {"pose": torch.cat([x[0] for x in done]).cpu().numpy(),
                "point": torch.cat([x[1] for x in done]).cpu().numpy(), "iterations": None}
    s = _BA(_graph(case, seed))
    if kind == "adapter":
        s.linearize()
        dx = s.solve(case["lam"])
        vec = lambda p, q: torch.cat([p[s.free].reshape(-1), q.reshape(-1)]).cpu().numpy()  # noqa: E731
        return {"b": vec(s.bp, s.bl), "x": vec(*dx)}
    _levenberg(s, case["iterations"])
    return {"pose": s.x[0].cpu().numpy(), "point": s.x[1].cpu().numpy(), "iterations": None}
