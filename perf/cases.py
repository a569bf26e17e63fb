"""The work that users of the library have it do, as cases that can be timed.

A case is a dict of plain values; its "kind" names the entry point that `run`
calls:

  solve     gba.solve on host arrays: the whole call, upload to download
  run       Solver.run from the starting parameters of a device-resident problem
  trial     one plain LM trial through the stage functions of a Solver
  linearize the normal equations and their damped point blocks at new parameters
  cholesky  dense_potrf and dense_potrs on device memory
  blocks    the batched 9x9 and 3x3 kernels
  edges     residuals and Jacobians (FP64 and FP32) and the allocation-free cost
  mlp       one training step of the coarse-basis network

Problems have the shapes of the library's synthetic workloads (power-law track
lengths, unit pixel noise, optional outliers, starting values off by a few per
cent); every size, and so the work of a pass, follows from the case alone, the
values from the seed.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "gpu-bundle-adjustment_gb300"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

MODEL = PACKAGE / "models" / "coarse_mlp.bin"
# Schur targets of the mixed forms: every step solved to the accuracy of the
# linearisation (the tightest that the library's tests ask for), so that two
# runs differ by far less than the steps
STRICT = {"refine_tol": 1e-10, "pcg_tol": 1e-4}
MLP_IN, MLP_USED_IN, MLP_H, MLP_OUT, MLP_USED_OUT = 64, 58, 128, 96, 81
MLP_SHAPES = ((MLP_H, MLP_IN), (MLP_H,), (MLP_H, MLP_H), (MLP_H,), (MLP_OUT, MLP_H), (MLP_OUT,))
ADAM = (1e-4, 0.9, 0.999, 1e-8)


def _solve(name, form, cameras, points, track_max, alpha, iterations, **more):
    return {"name": name, "kind": "solve", "form": form, "cameras": cameras, "points": points,
            "track_max": track_max, "alpha": alpha, "iterations": iterations, "window": 0, "huber": 0.0,
            "outliers": 0.0, "damping": 1e-2 if form == "mixed" else 1e-3, **more}


def listed():
    return [
        # a handful of images, the library's smallest workload: latency and launches count
        _solve("solve-plain-16", "plain", 16, 22000, 8, 1.29, 3),
        # a photo collection of a few hundred images, the default form, robust loss
        _solve("solve-plain-257", "plain", 257, 65000, 12, 2.23, 3, huber=2.0),
        # images along a path (a drive, a flight line): S is a band
        _solve("solve-plain-path-611", "plain", 611, 61003, 8, 1.5, 3, window=10),
        # one FP64 trial of a thousand images, stage by stage: the dense system of 9,000 unknowns
        {**_solve("trial-plain-1000", "plain", 1000, 200000, 16, 2.05, 1), "kind": "trial"},
        # the implicit form with block-Jacobi, tight Schur targets
        _solve("solve-mixed-1000", "mixed", 1000, 200000, 16, 2.05, 2),
        # a collection like the plain form's second case with the learned coarse space
        _solve("solve-learned-257", "learned", 257, 65000, 12, 2.23, 2),
        # the benchmark's workload: 5,000 images, 8.8 million observations, 5 % outliers
        {**_solve("run-learned-5000", "learned", 5000, 1500000, 200, 2.2, 2, outliers=0.05), "kind": "run"},
        # FP32 Jacobians and normal equations of a large problem, for callers that drive the stages
        {**_solve("linearize-mixed-2477", "mixed", 2477, 611003, 60, 2.1, 1, outliers=0.05), "kind": "linearize"},
        # the dense factorisation and solve for callers that assemble their own system
        {"name": "cholesky-4096", "kind": "cholesky", "n": 4096},
        # camera and point blocks of a mid-sized problem
        {"name": "blocks-5003", "kind": "blocks", "n9": 5003, "n3": 200003},
        # residuals, Jacobians and cost of 800,000 observations for callers with their own solver
        {"name": "edges-800335", "kind": "edges", "cameras": 1000, "points": 200000, "edges": 800335},
        # a training step of the coarse-basis network on one system
        {"name": "mlp-1000", "kind": "mlp", "batch": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "path", "trial", "mixed", "learned", "run", "linearize", "cholesky", "blocks",
                       "edges", "mlp"])
    alpha = round(rng.uniform(1.3, 2.4), 3)
    huber = rng.choice([0.0, round(rng.uniform(0.8, 4.0), 2)])
    if kind == "plain":
        cameras = _log(rng, 9, 400)
        case = _solve("", "plain", cameras, _log(rng, 3000, 90000), min(cameras, rng.randint(4, 12)), alpha,
                      rng.randint(2, 3), huber=huber)
    elif kind == "path":
        cameras = _log(rng, 90, 800)
        case = _solve("", "plain", cameras, rng.randint(60, 120) * cameras + rng.randint(0, 63), rng.randint(4, 9),
                      alpha, rng.randint(2, 3), window=rng.randint(5, 12), huber=huber)
    elif kind == "trial":
        cameras = _log(rng, 200, 1000)
        case = {**_solve("", "plain", cameras, 200 * cameras - rng.randint(0, 99), rng.randint(6, 16), 2.05, 1),
                "kind": "trial"}
    elif kind in ("mixed", "learned"):
        cameras = _log(rng, 33, 1000)
        case = _solve("", kind, cameras, max(20000, 200 * cameras) + rng.randint(0, 999), rng.randint(6, 24), alpha,
                      2, huber=huber)
    elif kind == "run":
        cameras = _log(rng, 600, 4000)
        case = {**_solve("", "learned", cameras, 250 * cameras + rng.randint(0, 999),
                         rng.randint(20, 200), round(rng.uniform(2.0, 2.4), 3), 2, outliers=0.05), "kind": "run"}
    elif kind == "linearize":
        cameras = _log(rng, 33, 4000)
        case = {**_solve("", rng.choice(["plain", "mixed"]), cameras, 200 * cameras + rng.randint(0, 999),
                         min(cameras, rng.randint(6, 100)), round(rng.uniform(2.0, 2.4), 3), 1, huber=huber),
                "kind": "linearize"}
    elif kind == "cholesky":
        case = {"kind": "cholesky", "n": 64 * _log(rng, 2, 64)}
    elif kind == "blocks":
        case = {"kind": "blocks", "n9": _log(rng, 50, 20000), "n3": _log(rng, 500, 1500000)}
    elif kind == "edges":
        edges = _log(rng, 3000, 2000000)
        case = {"kind": "edges", "cameras": max(8, edges // 900), "points": max(100, edges // 4), "edges": edges}
    else:
        case = {"kind": "mlp", "batch": _log(rng, 16, 5000)}
    case.pop("name", None)
    return case


# ---------------------------------------------------------------- inputs

def _tracks(case):
    """Track lengths of the case's points (sorted): a power law over [2, track_max]."""
    k = np.arange(2, max(2, case["track_max"]) + 1, dtype=np.float64)
    cdf = np.cumsum(k ** -case["alpha"])
    at = (np.arange(case["points"]) + 0.5) / case["points"] * cdf[-1]
    return 2 + np.minimum(np.searchsorted(cdf, at), k.size - 1)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _project(cams, pts):
    """Predicted pixels and the pieces of the camera model (rows of cams and pts in pairs)."""
    a, t = cams[:, 0:3], cams[:, 3:6]
    f, k1, k2 = cams[:, 6], cams[:, 7], cams[:, 8]
    th = a.norm(dim=1, keepdim=True).clamp_min(1e-300)
    w = a / th
    s, omc = torch.sin(th), 2.0 * torch.sin(0.5 * th) ** 2
    RX = (1.0 - omc) * pts + s * torch.linalg.cross(w, pts) + omc * (w * pts).sum(1, keepdim=True) * w
    X = RX + t
    u, v = -X[:, 0] / X[:, 2], -X[:, 1] / X[:, 2]
    r2 = u * u + v * v
    d = 1.0 + r2 * (k1 + k2 * r2)
    return torch.stack((f * d * u, f * d * v), 1), (w, th, s, omc, RX, X, u, v, r2, d)


def _cameras(g, n):
    """Cameras on a ring of radius 1.5, looking at points some four to ten units away."""
    c = torch.empty(n, 9, device="cuda", dtype=torch.float64)
    at = 2.0 * math.pi / n * torch.arange(n, device="cuda", dtype=torch.float64)
    c[:, 0:3] = 0.1 * _normal(g, n, 3)
    c[:, 3:6] = torch.stack((1.5 * at.cos(), 1.5 * at.sin(), _uniform(g, -0.3, 0.3, n)), 1)
    c[:, 6] = _uniform(g, 400.0, 600.0, n)
    c[:, 7] = 1e-2 * _normal(g, n)
    c[:, 8] = 1e-4 * _normal(g, n)
    return c


def _rotate(cams, x):
    """R(a) x for each camera's angle-axis a."""
    still = cams.clone()
    still[:, 3:6] = 0.0
    return _project(still, x)[1][4]


def _problem(case, seed):
    """A seeded problem: (cameras, points, obs_camera, obs_point, obs_pixel) on the GPU."""
    g = _generator(seed)
    C, P, window = case["cameras"], case["points"], case["window"]
    true_cams = _cameras(g, C)
    pts = torch.stack((_uniform(g, -3.0, 3.0, P), _uniform(g, -3.0, 3.0, P), _uniform(g, -10.0, -4.0, P)), 1)
    centre = None
    if window:  # cameras half a unit apart along x, points beside the path
        centre = 0.1 * _normal(g, C, 3)
        centre[:, 0] = 0.5 * torch.arange(C, device="cuda", dtype=torch.float64)
        true_cams[:, 3:6] = -_rotate(true_cams, centre)
        pts[:, 0] = _uniform(g, -1.0, 0.5 * (C - 1) + 1.0, P)
    k = torch.from_numpy(_tracks(case)).cuda()[torch.randperm(P, generator=g, device="cuda")]
    # distinct cameras for each point: an arithmetic progression of random
    # start and step modulo the cameras that can see it (steps prime to them,
    # and at least an eighth of them, so that two views have a baseline)
    near = min(C, 2 * window + 1) if window else C
    first = torch.zeros(P, device="cuda", dtype=torch.int64)
    if window:
        first = ((pts[:, 0] / 0.5).round().long() - window).clamp(0, C - near)
    steps = torch.tensor([s for s in range(1, near) if math.gcd(s, near) == 1 and near <= 8 * s <= 7 * near] or [1],
                         device="cuda")
    start = torch.randint(near, (P,), generator=g, device="cuda")
    step = steps[torch.randint(steps.numel(), (P,), generator=g, device="cuda")]
    k = k.clamp(max=near)
    op = torch.repeat_interleave(torch.arange(P, device="cuda"), k)
    j = torch.arange(op.numel(), device="cuda") - torch.repeat_interleave(k.cumsum(0) - k, k)
    oc = first[op] + (start[op] + j * step[op]) % near
    by_camera = torch.argsort(oc, stable=True)
    oc, op = oc[by_camera], op[by_camera]
    E = oc.numel()
    sigma = torch.where(torch.rand(E, 1, generator=g, device="cuda") < case["outliers"], 20.0, 1.0)
    px = _project(true_cams[oc], pts[op])[0] + sigma * _normal(g, E, 2)
    cams = true_cams + 0.01 * _normal(g, C, 9)
    if window:  # rotations and centres are off, not the translation that grows along the path
        cams[:, 3:6] = -_rotate(cams, centre + 0.01 * _normal(g, C, 3))
    return cams, pts + 0.05 * _normal(g, P, 3), oc.int(), op.int(), px


def _options(case):
    o = {"form": case["form"], "max_iterations": case["iterations"], "initial_lambda": case["damping"]}
    if case["form"] != "plain":
        o.update(STRICT)
    if case["form"] == "learned":
        o["model_path"] = MODEL
    if case["huber"] > 0.0:
        o.update(loss="huber", huber_delta=case["huber"])
    return o


class _View:
    """A buffer of a solver as the array interface that torch reads; the tensor keeps the solver alive."""

    def __init__(self, solver, name, n):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (solver.device_ptr(name), False),
                                         "version": 3}


def _view(solver, name, n):
    return torch.as_tensor(_View(solver, name, n), device="cuda")


def _spd_system(n, seed):
    """An SPD matrix with the scale spread of a reduced camera system, and a right-hand side."""
    g = _generator(seed)
    scale = torch.tensor([3.0, 3.0, 2.0, 1.0, 1.0, 0.5, 0.02, 5.0, 8.0], device="cuda", dtype=torch.float64)
    d = scale.repeat(n // 9 + 1)[:n] * torch.exp(0.3 * _normal(g, n))
    B = _normal(g, n, max(64, n // 2))
    A = (B @ B.T) / B.shape[1]
    A.diagonal().add_(0.3)
    return A * d[:, None] * d[None, :], d * _normal(g, n)


def _spd_blocks(g, n, m):
    B = _normal(g, n, m, m)
    return B @ B.transpose(1, 2) + 0.1 * torch.eye(m, device="cuda", dtype=torch.float64)


def _mlp_params(g):
    parts = []
    for shape in MLP_SHAPES:
        if len(shape) == 2:
            parts.append(_normal(g, *shape).mul_(math.sqrt(2.0 / shape[1])).reshape(-1))
        else:
            parts.append(0.1 * _normal(g, *shape))
    parts[4] = 0.1 * parts[4]
    return torch.cat(parts).float()


def _mlp_batch(case, seed):
    g = _generator(seed)
    B = case["batch"]
    params = _mlp_params(g)
    feat = torch.zeros(B, MLP_IN, device="cuda")
    feat[:, :MLP_USED_IN] = (0.5 * _normal(g, B, MLP_USED_IN)).float()
    grad = torch.zeros(B, MLP_OUT, device="cuda")
    grad[:, :MLP_USED_OUT] = (1e-2 * _normal(g, B, MLP_USED_OUT)).float()
    return params, feat, grad


def _edges(case, seed):
    g = _generator(seed)
    E = case["edges"]
    cams = _cameras(g, case["cameras"])
    P = case["points"]
    pts = torch.stack((_uniform(g, -3.0, 3.0, P), _uniform(g, -3.0, 3.0, P), _uniform(g, -10.0, -4.0, P)), 1)
    oc = torch.randint(case["cameras"], (E,), generator=g, device="cuda")
    op = torch.randint(P, (E,), generator=g, device="cuda")
    px = _project(cams[oc], pts[op])[0] + _normal(g, E, 2)
    return cams, pts, oc.int(), op.int(), px


def _host_problem(gba, case, seed):
    cams, pts, oc, op, px = (t.cpu().numpy().reshape(-1) for t in _problem(case, seed))
    return gba.BALProblem(cams, pts, oc, op, px)


def prepare(case, seed):
    import gba_gb300 as gba

    s = {"gba": gba, "case": case}
    kind = case["kind"]
    if kind == "solve":
        s["problem"] = _host_problem(gba, case, seed)
        s["options"] = _options(case)
    elif kind in ("run", "trial", "linearize"):
        problem = _host_problem(gba, case, seed)
        s["solver"] = gba.Solver(problem, case["form"])
        s["sizes"] = problem.cameras.size, problem.points.size
        s["options"] = _options(case)
        if kind != "run" and case["huber"] > 0.0:
            s["solver"].set_loss("huber", case["huber"])
        if case["form"] == "learned":
            s["solver"].load_model(MODEL)
            s["options"].pop("model_path")
    elif kind == "cholesky":
        s["A"], s["b"] = _spd_system(case["n"], seed)
        s["L"], s["x"] = torch.empty_like(s["A"]), torch.empty_like(s["b"])
        s["info"] = torch.zeros(1, device="cuda", dtype=torch.int32)
    elif kind == "blocks":
        g = _generator(seed)
        s["A9"], s["b9"] = _spd_blocks(g, case["n9"], 9), _normal(g, case["n9"], 9)
        s["A3"] = _spd_blocks(g, case["n3"], 3)
        s["x9"], s["inv3"] = torch.empty_like(s["b9"]), torch.empty_like(s["A3"])
        s["ok9"] = torch.zeros(case["n9"], device="cuda", dtype=torch.int32)
        s["ok3"] = torch.zeros(case["n3"], device="cuda", dtype=torch.int32)
    elif kind == "edges":
        s["in"] = tuple(t.contiguous() for t in _edges(case, seed))
        for name, t in (("64", torch.float64), ("32", torch.float32)):
            for part, n in (("r", 2), ("jc", 18), ("jp", 6)):
                s[part + name] = torch.empty(case["edges"], n, device="cuda", dtype=t)
        s["sse"] = torch.empty(1, device="cuda", dtype=torch.float64)
        s["bad"] = torch.zeros(1, device="cuda", dtype=torch.int64)
    else:
        params, s["feat"], s["grad"] = _mlp_batch(case, seed)
        s["mlp"] = gba.Mlp(seed=0, capacity=case["batch"])
        s["mlp"].set_params(params.cpu().numpy())
        s["out"] = torch.empty(case["batch"], MLP_OUT, device="cuda")
    return s


def run(s):
    gba, kind = s["gba"], s["case"]["kind"]
    if kind == "solve":
        p = s["problem"]
        p = gba.BALProblem(p.cameras.copy(), p.points.copy(), p.obs_camera, p.obs_point, p.obs_pixel)
        res = gba.solve(p, **s["options"])
        return {"cameras": p.cameras, "points": p.points, "trajectory": np.array(res.trajectory)}
    if kind == "run":
        solver, (nc, np_) = s["solver"], s["sizes"]
        solver.reset_params()
        res = solver.run(**s["options"])
        return {"cameras": _view(solver, "cams", nc), "points": _view(solver, "pts", np_),
                "trajectory": np.array(res.trajectory)}
    if kind == "trial":
        solver, (nc, np_), lam = s["solver"], s["sizes"], s["case"]["damping"]
        sse = solver.accumulate()
        bad = solver.damp_invert_v(lam)
        info = solver.schur_dense(lam)
        denom = solver.back_substitute(lam)
        return {"sse": sse, "bad": bad, "info": info, "denominator": denom, "trial_sse": solver.trial_cost(),
                "dc": _view(solver, "dc", nc), "dp": _view(solver, "dp", np_)}
    if kind == "linearize":
        solver, (nc, np_) = s["solver"], s["sizes"]
        solver.reset_params()
        return {"sse": solver.accumulate(), "bad": solver.damp_invert_v(s["case"]["damping"]),
                "U": _view(solver, "U", 9 * nc), "V": _view(solver, "V", 2 * np_), "bc": _view(solver, "bc", nc), "bp": _view(solver, "bp", np_)}
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "cholesky":
        n, L, x, info = s["case"]["n"], s["L"], s["x"], s["info"]
        L.copy_(s["A"])
        x.copy_(s["b"])
        gba.dense_potrf(L.data_ptr(), n, n, info.data_ptr(), stream)
        gba.dense_potrs(L.data_ptr(), n, n, x.data_ptr(), info.data_ptr(), stream)
        # column-major lower triangle: the upper one of the row-major tensor
        return {"factor": torch.triu(L), "x": x, "info": info}
    if kind == "blocks":
        gba.batch_chol9_factor_solve(s["A9"].data_ptr(), s["b9"].data_ptr(), s["x9"].data_ptr(), s["ok9"].data_ptr(),
                                     s["case"]["n9"], stream)
        gba.batch_inverse3_spd(s["A3"].data_ptr(), s["inv3"].data_ptr(), s["ok3"].data_ptr(), s["case"]["n3"], stream)
        return {"x9": s["x9"], "ok9": s["ok9"], "inv3": s["inv3"], "ok3": s["ok3"]}
    if kind == "edges":
        E = s["case"]["edges"]
        at = [t.data_ptr() for t in s["in"]]
        for precision, name in ((64, "64"), (32, "32")):
            gba.eval_edges(precision, *at, E, s["r" + name].data_ptr(), s["jc" + name].data_ptr(),
                           s["jp" + name].data_ptr(), stream)
        status = gba.lib.gba_cost_noalloc(*at, E, s["sse"].data_ptr(), s["bad"].data_ptr(), stream or None)
        return {**{k: s[k] for k in ("r64", "jc64", "jp64", "r32", "jc32", "jp32", "sse", "bad")}, "status": status}
    mlp, B = s["mlp"], s["case"]["batch"]
    mlp.forward(s["feat"].data_ptr(), B, s["out"].data_ptr(), stream)
    mlp.backward(s["feat"].data_ptr(), s["grad"].data_ptr(), B, stream)
    mlp.adam_step(*ADAM, stream=stream)
    return {"out": s["out"], "grads": mlp.grads(), "params": mlp.params()}


# ---------------------------------------------------------------- work

def work(case):
    kind = case["kind"]
    if kind == "cholesky":
        n = case["n"]
        return {"bytes": 8.0 * n * (n + 1), "flops": n ** 3 / 3.0 + 2.0 * n * n}
    if kind == "blocks":
        return {"bytes": 8.0 * (case["n9"] * 99 + case["n3"] * 18) + 4.0 * (case["n9"] + case["n3"]),
                "flops": 450.0 * case["n9"] + 60.0 * case["n3"]}
    if kind == "edges":
        E, C, P = case["edges"], case["cameras"], case["points"]
        return {"bytes": 24.0 * E + 72.0 * C + 24.0 * P + 26 * 12.0 * E, "flops": 500.0 * E}
    if kind == "mlp":
        weights = sum(int(np.prod(s)) for s in MLP_SHAPES)
        return {"bytes": 4.0 * case["batch"] * (MLP_IN + 2 * MLP_OUT) + 4.0 * 8 * weights,
                "flops": 5.0 * case["batch"] * weights}
    k = _tracks(case).astype(np.float64)
    C, P, E, T = case["cameras"], case["points"], float(k.sum()), case["iterations"]
    bytes_ = 24.0 * E + 2 * (72.0 * C + 24.0 * P)
    flops = T * E * 700.0
    if kind == "linearize":  # the parameters and observations in; U, V, bc, bp and the Jacobians out
        jacobians = (27 + 20) * 8.0 if case["form"] == "plain" else 24 * 4.0
        return {"bytes": 24.0 * E + 72.0 * C + 24.0 * P + 720.0 * C + 72.0 * P + jacobians * E, "flops": flops}
    if case["form"] == "plain":
        n = 9.0 * C
        width = min(n, 9.0 * (2 * case["window"] + 1)) if case["window"] else 0.0
        flops += T * (243.0 * float((k * (k + 1)).sum()) + (n * width * width if width else n ** 3 / 3.0))
    else:  # three inner solves a step of at least ten products
        flops += T * 30 * E * 100.0
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------- 64-bit results

def _jacobian(cams, pts):
    """Predicted pixels, and their derivatives by the camera (E, 2, 9) and the point (E, 2, 3)."""
    pred, (w, th, s, omc, RX, X, u, v, r2, d) = _project(cams, pts)
    f, k1, k2 = cams[:, 6], cams[:, 7], cams[:, 8]
    E = cams.shape[0]
    one, zero = torch.ones_like(u), torch.zeros_like(u)
    L = k1 + 2.0 * k2 * r2
    uv = torch.stack((u, v), 1)
    D = (f * d)[:, None, None] * torch.eye(2, device=u.device, dtype=u.dtype) \
        + (2.0 * f * L)[:, None, None] * uv[:, :, None] * uv[:, None, :]
    iz = 1.0 / X[:, 2]
    M = torch.stack((torch.stack((-one, zero, -u), 1), torch.stack((zero, -one, -v), 1)), 1) * iz[:, None, None]
    G = D @ M

    def skew(x):
        z = torch.zeros_like(x[:, 0])
        return torch.stack((z, -x[:, 2], x[:, 1], x[:, 2], z, -x[:, 0], -x[:, 1], x[:, 0], z), 1).reshape(E, 3, 3)

    eye = torch.eye(3, device=u.device, dtype=u.dtype)
    K, ww = skew(w), w[:, :, None] * w[:, None, :]
    s, omc, th = s[:, :, None], omc[:, :, None], th[:, :, None]
    R = (1.0 - omc) * eye + s * K + omc * ww
    Jl = (s / th) * eye + (omc / th) * K + (1.0 - s / th) * ww
    Jc = torch.cat((-(G @ skew(RX)) @ Jl, G, (d[:, None] * uv)[:, :, None], ((f * r2)[:, None] * uv)[:, :, None],
                    ((f * r2 * r2)[:, None] * uv)[:, :, None]), 2)
    return pred, Jc, G @ R


class _Exact:
    """The plain Levenberg-Marquardt iteration in FP64 torch operations."""

    def __init__(self, case, seed):
        cams, pts, oc, op, self.px = _problem(case, seed)
        self.cams, self.pts, self.oc, self.op = cams, pts, oc.long(), op.long()
        self.delta, self.damping = case["huber"], case["damping"]
        self.C, self.P = case["cameras"], case["points"]
        order = torch.argsort(self.op, stable=True)
        counts = torch.bincount(self.op, minlength=self.P)
        begin = counts.cumsum(0) - counts
        self.groups = []  # observations of the points of each track length, (points, length)
        for k in range(1, int(counts.max()) + 1):
            p = (counts == k).nonzero()[:, 0]
            if p.numel():
                self.groups.append((p, order[begin[p][:, None] + torch.arange(k, device="cuda")]))

    def cost(self, cams, pts):
        r = _project(cams[self.oc], pts[self.op])[0] - self.px
        return self._rho(r.square().sum(1)).sum().item()

    def _rho(self, s):
        if self.delta <= 0.0:
            return s
        return torch.where(s > self.delta ** 2, 2.0 * self.delta * s.sqrt() - self.delta ** 2, s)

    def normal_equations(self):
        pred, Jc, Jp = _jacobian(self.cams[self.oc], self.pts[self.op])
        r = pred - self.px
        s = r.square().sum(1)
        sse = self._rho(s).sum().item()
        if self.delta > 0.0:
            w = torch.where(s > self.delta ** 2, (self.delta / s.sqrt()).sqrt(), torch.ones_like(s))
            r, Jc, Jp = r * w[:, None], Jc * w[:, None, None], Jp * w[:, None, None]
        add = lambda n, i, v: torch.zeros(n, *v.shape[1:], device="cuda", dtype=v.dtype).index_add_(0, i, v)  # noqa: E731
        Jct, Jpt = Jc.transpose(1, 2), Jp.transpose(1, 2)
        self.U, self.V = add(self.C, self.oc, Jct @ Jc), add(self.P, self.op, Jpt @ Jp)
        self.bc = -add(self.C, self.oc, (Jct @ r[:, :, None])[:, :, 0])
        self.bp = -add(self.P, self.op, (Jpt @ r[:, :, None])[:, :, 0])
        self.W = Jct @ Jp
        return sse

    @staticmethod
    def _damp(B, lam):
        d = B.diagonal(dim1=1, dim2=2)
        return B + torch.diag_embed(lam * torch.where(d > 0.0, d, torch.full_like(d, 1e-12)))

    def step(self, lam):
        C, n = self.C, 9 * self.C
        Vi = torch.linalg.inv(self._damp(self.V, lam))
        S = torch.zeros(C * C, 81, device="cuda", dtype=torch.float64)
        rhs = self.bc.clone()
        for p, e in self.groups:
            k = e.shape[1]
            room = max(1, 2_000_000 // (k * k))
            for i in range(0, p.numel(), room):
                q, f = p[i:i + room], e[i:i + room]
                W = self.W[f]
                T = W @ Vi[q][:, None]
                B = T[:, :, None] @ W[:, None].transpose(3, 4)
                c = self.oc[f]
                S.index_add_(0, (c[:, :, None] * C + c[:, None, :]).reshape(-1), B.reshape(-1, 81), alpha=-1.0)
                rhs.index_add_(0, c.reshape(-1), (T @ self.bp[q][:, None, :, None])[..., 0].reshape(-1, 9), alpha=-1.0)
        at = torch.arange(C, device="cuda") * (C + 1)
        S[at] += self._damp(self.U, lam).reshape(C, 81)
        S = S.reshape(C, C, 9, 9).permute(0, 2, 1, 3).reshape(n, n)
        L, info = torch.linalg.cholesky_ex(0.5 * (S + S.T))
        if int(info):
            return None
        dc = torch.cholesky_solve(rhs.reshape(n, 1), L).reshape(C, 9)
        back = torch.zeros_like(self.bp).index_add_(0, self.op, (self.W.transpose(1, 2) @ dc[self.oc][:, :, None])[:, :, 0])
        dp = (Vi @ (self.bp - back)[:, :, None])[:, :, 0]
        denom = 0.0
        for x, B, b in ((dc, self.U, self.bc), (dp, self.V, self.bp)):
            d = B.diagonal(dim1=1, dim2=2)
            denom += (x * (lam * torch.where(d > 0.0, d, torch.full_like(d, 1e-12)) * x + b)).sum().item()
        return dc, dp, denom

    def solve(self, iterations):
        sse, lam, trajectory = self.normal_equations(), self.damping, []
        trajectory.append(sse / 2.0)
        for _ in range(iterations):
            nu, accepted, gain = 2.0, False, 0.0
            for _ in range(16):
                got = self.step(lam)
                if got and got[2] > 0.0:
                    dc, dp, denom = got
                    trial = self.cost(self.cams + dc, self.pts + dp)
                    rho = (sse - trial) / (0.5 * denom)
                    if rho > 0.0 and trial < sse:
                        self.cams, self.pts = self.cams + dc, self.pts + dp
                        gain, sse, accepted = (sse - trial) / max(sse, 1.0), trial, True
                        lam *= max(1.0 / 3.0, 1.0 - (2.0 * rho - 1.0) ** 3)
                        break
                lam, nu = lam * nu, nu * 2.0
            if not accepted:
                break
            trajectory.append(sse / 2.0)
            if gain < 1e-6:
                break
            self.normal_equations()
        return {"cameras": self.cams.reshape(-1), "points": self.pts.reshape(-1), "trajectory": np.array(trajectory)}


def _exact_mlp(case, seed):
    params, feat, grad = (t.double() for t in _mlp_batch(case, seed))
    W, at = [], 0
    for shape in MLP_SHAPES:
        W.append(params[at:at + int(np.prod(shape))].reshape(shape))
        at += int(np.prod(shape))
    h1 = (feat @ W[0].T + W[1]).clamp_min(0.0)
    h2 = (h1 @ W[2].T + W[3]).clamp_min(0.0)
    out = h2 @ W[4].T + W[5]
    d2 = (grad @ W[4]) * (h2 > 0.0)
    d1 = (d2 @ W[2]) * (h1 > 0.0)
    grads = torch.cat([t.reshape(-1) for t in (d1.T @ feat, d1.sum(0), d2.T @ h1, d2.sum(0), grad.T @ h2, grad.sum(0))])
    lr, _, _, eps = ADAM
    new = params - lr * grads / (grads.abs() + eps)  # the first step: both moments are the gradient's own
    return {"out": out, "grads": grads, "params": new}


def exact(case, seed):
    kind = case["kind"]
    if kind == "cholesky":
        A, b = _spd_system(case["n"], seed)
        L = torch.linalg.cholesky(A)
        return {"factor": L.T.contiguous(), "x": torch.cholesky_solve(b[:, None], L)[:, 0], "info": None}
    if kind == "blocks":
        g = _generator(seed)
        A9, b9 = _spd_blocks(g, case["n9"], 9), _normal(g, case["n9"], 9)
        return {"x9": torch.linalg.solve(A9, b9), "ok9": None, "inv3": torch.linalg.inv(_spd_blocks(g, case["n3"], 3)),
                "ok3": None}
    if kind == "edges":
        cams, pts, oc, op, px = _edges(case, seed)
        pred, Jc, Jp = _jacobian(cams[oc.long()], pts[op.long()])
        r, Jc, Jp = pred - px, Jc.reshape(-1, 18), Jp.reshape(-1, 6)
        return {"r64": r, "jc64": Jc, "jp64": Jp, "r32": r, "jc32": Jc, "jp32": Jp,
                "sse": r.square().sum().reshape(1), "bad": None, "status": None}
    if kind == "mlp":
        return _exact_mlp(case, seed)
    if case["cameras"] > 1100 and kind != "linearize":  # a dense system too large for this
        return None
    e = _Exact(case, seed)
    if kind == "linearize":
        sse, tril = e.normal_equations(), torch.tril_indices(3, 3, device="cuda")
        return {"sse": sse, "bad": None, "U": e.U.reshape(-1), "V": e.V[:, tril[0], tril[1]].reshape(-1),
                "bc": e.bc.reshape(-1), "bp": e.bp.reshape(-1)}
    if kind == "trial":
        sse = e.normal_equations()
        dc, dp, denom = e.step(case["damping"])
        return {"sse": sse, "bad": None, "info": None, "denominator": denom,
                "trial_sse": e.cost(e.cams + dc, e.pts + dp), "dc": dc.reshape(-1), "dp": dp.reshape(-1)}
    return e.solve(case["iterations"])
