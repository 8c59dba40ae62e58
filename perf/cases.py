"""The work that is timed: evaluations of the dual functional and its gradient (single problems, batches,
truncated and untruncated, hexahedral and simplex sources, both precision modes), the tensor-core Hessian and
the L-BFGS solve, each through the public entry points of ``semidiscreteot_b200``.

A case is a dict of plain values:

  kind     "dense" | "tet" | "trunc" | "hessian" | "batch" | "solve"
  dim      2 or 3
  side     cells per axis of the structured mesh (cubes per axis of the tetrahedral mesh)
  order    Gauss points per axis of a cell (simplex rules: 1, 2, 3)
  targets  number of targets
  eps      entropic regularisation
  prec     "hybrid" (the default: FP64 values, FP32 exponentials in the gradient) | "fp64" (what the Newton
           and the tight solves run on)
  host     True: potentials and gradients are host arrays; False: device tensors
"""
from __future__ import annotations

import math

import numpy as np
import torch

from semidiscreteot_b200 import BatchSolver, SolverParameters, SotSolver, simplex_source, structured_source
from semidiscreteot_b200.simplex import tetra_cube_mesh

TAU = 1e-12          # truncation tolerance of the truncated problems
SOLVE_STEPS = 10     # L-BFGS iterations of the solve


def listed():
    return [
        # one small problem of a batch or of a coarse level: 2,304 points, launches and latency count
        {"name": "dense_2d_small", "kind": "dense", "dim": 2, "side": 16, "order": 3, "targets": 256, "eps": 1e-1,
         "prec": "hybrid", "host": False},
        # the dense benchmark problem (64 x 64 cells, QGauss(3), 1,000 targets) as a host program calls it
        {"name": "dense_2d", "kind": "dense", "dim": 2, "side": 64, "order": 3, "targets": 1000, "eps": 1e-2,
         "prec": "hybrid", "host": True},
        # a ragged mid-size problem in the precision of a tight solve: order 2, odd side and count
        {"name": "dense_2d_odd_fp64", "kind": "dense", "dim": 2, "side": 75, "order": 2, "targets": 3001, "eps": 1e-2,
         "prec": "fp64", "host": False},
        # the largest problem of the batched configuration (128 x 128 cells, 16,384 targets, smallest eps)
        {"name": "dense_2d_large", "kind": "dense", "dim": 2, "side": 128, "order": 3, "targets": 16384, "eps": 1e-3,
         "prec": "hybrid", "host": False},
        # the evaluation inside the Newton configuration (32^3 hexahedra, 20,000 targets)
        {"name": "dense_3d_fp64", "kind": "dense", "dim": 3, "side": 32, "order": 2, "targets": 20000, "eps": 5e-3,
         "prec": "fp64", "host": False},
        # a tetrahedral source without any grid structure, as the first tutorial's
        {"name": "tet_3d", "kind": "tet", "dim": 3, "side": 8, "order": 3, "targets": 1000, "eps": 1e-2,
         "prec": "hybrid", "host": False},
        # the headline benchmark: 64^3 hexahedra, 100,000 clustered targets, truncated
        {"name": "trunc_3d", "kind": "trunc", "dim": 3, "side": 64, "order": 2, "targets": 100000, "eps": 1e-3,
         "prec": "hybrid", "host": False},
        # the same at a ragged eighth of its size, from host arrays
        {"name": "trunc_3d_odd", "kind": "trunc", "dim": 3, "side": 31, "order": 2, "targets": 12345, "eps": 1e-3,
         "prec": "hybrid", "host": True},
        # a truncated problem in the plane, in the precision of a tight solve
        {"name": "trunc_2d_fp64", "kind": "trunc", "dim": 2, "side": 128, "order": 3, "targets": 10000, "eps": 1e-4,
         "prec": "fp64", "host": False},
        # the Hessian of the Newton configuration, FP32 entries as Newton keeps them
        {"name": "hessian_3d", "kind": "hessian", "dim": 3, "side": 32, "order": 2, "targets": 20000, "eps": 5e-3,
         "prec": "fp64", "host": False},
        # one evaluation of a batch of uneven problems (every round of a batched solve is one)
        {"name": "batch_2d", "kind": "batch", "dim": 2, "side": 128, "order": 3, "targets": 16384, "eps": 1e-3,
         "prec": "fp64", "host": True, "problems": 16},
        # the first iterations of an L-BFGS solve: evaluations, the two-loop recursion and the line search
        {"name": "solve_2d", "kind": "solve", "dim": 2, "side": 32, "order": 3, "targets": 500, "eps": 5e-2,
         "prec": "fp64", "host": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "tet", "trunc", "trunc", "hessian", "batch", "solve"])
    prec = rng.choice(["hybrid", "fp64"])
    c = {"kind": kind, "dim": 2, "order": 3, "prec": prec, "host": rng.random() < 0.3}
    if kind == "dense":
        c["dim"] = rng.choice([2, 3])
        if c["dim"] == 2:
            c.update(side=_log(rng, 8, 128), order=rng.choice([2, 3]), targets=_log(rng, 64, 16384),
                     eps=rng.choice([1e-1, 1e-2, 1e-3]))
        else:
            c.update(side=_log(rng, 6, 32), order=2, targets=_log(rng, 100, 20000), eps=rng.choice([1e-2, 5e-3]))
    elif kind == "tet":
        c.update(dim=3, side=_log(rng, 3, 8), order=rng.choice([2, 3]), targets=_log(rng, 100, 2000), eps=1e-2)
    elif kind == "trunc":
        c["dim"] = rng.choice([2, 3])
        if c["dim"] == 2:
            c.update(side=_log(rng, 32, 128), order=rng.choice([2, 3]), targets=_log(rng, 1000, 10000),
                     eps=rng.choice([1e-3, 1e-4]))
        else:
            c.update(side=_log(rng, 16, 64), order=2, targets=_log(rng, 2000, 100000), eps=1e-3)
    elif kind == "hessian":
        c.update(dim=3, side=_log(rng, 8, 32), order=2, targets=_log(rng, 300, 20000), eps=rng.choice([1e-2, 5e-3]),
                 prec="fp64", host=False)
    elif kind == "batch":
        c.update(side=_log(rng, 32, 128), targets=_log(rng, 1024, 16384), eps=rng.choice([1e-1, 1e-2, 1e-3]),
                 host=True, problems=rng.randint(4, 24))
    else:
        c.update(side=_log(rng, 12, 64), targets=_log(rng, 100, 2000), eps=rng.choice([1e-1, 5e-2]), prec="fp64",
                 host=True)
    return c


# ---------------------------------------------------------------------------------------------------- inputs

def _bumps(rng, dim):
    """A density made of a few Gaussian bumps on a floor."""
    k = int(rng.integers(2, 5))
    mu, sig, amp = rng.uniform(0.15, 0.85, (k, dim)), rng.uniform(0.08, 0.3, k), rng.uniform(0.5, 2.0, k)

    def density(p):
        out = np.full(p.shape[0], 0.05)
        for m, s, a in zip(mu, sig, amp):
            out += a * np.exp(-0.5 * np.sum((p - m) ** 2, axis=1) / s ** 2)
        return out

    return density


def _problem(kind, dim, side, order, targets, eps, rng):
    """Source, targets, weights and a potential of a solve under way (a smooth part and noise, a few eps high)."""
    if kind == "tet":
        vertices, cells = tetra_cube_mesh(side, 0.0, 1.0)
        src = simplex_source(vertices, cells, _bumps(rng, dim), order=order)
    else:
        src = structured_source(dim, side, order, nodal_density=_bumps(rng, dim))
    if kind == "trunc":   # clustered targets
        means, sig = rng.uniform(0.1, 0.9, (6, dim)), rng.uniform(0.05, 0.2, 6)
        comp = rng.choice(6, size=targets, p=rng.dirichlet(np.ones(6)))
        y = np.clip(means[comp] + rng.standard_normal((targets, dim)) * sig[comp, None], 0.0, 1.0)
    else:
        y = rng.random((targets, dim))
    # weights of Dirichlet(1) type, no smaller than a thousandth of the mean
    nu = rng.standard_exponential(targets) + 1e-3
    nu /= nu.sum()
    phase = rng.uniform(0.0, 2.0 * np.pi, dim)
    psi = eps * (np.sum(np.sin(2.0 * np.pi * y + phase), axis=1) / dim + 0.3 * rng.standard_normal(targets))
    return src, y, nu, psi - psi.mean()


def _batch_sizes(case):
    """(side, targets, eps) of the problems: spread over the logarithm of the sizes, up to the case's own."""
    n, out = case["problems"], []
    for i in range(n):
        u, v = (i + 0.5) / n, (i * 0.6180339887498949 + 0.5) % 1.0
        side = int(round(16 * (case["side"] / 16) ** u))
        targets = int(round(256 * (case["targets"] / 256) ** v))
        out.append((side, targets, (1e-1, 1e-2, case["eps"])[i % 3]))
    return out


def _problems(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        return [(s, t, e, _problem("dense", case["dim"], s, case["order"], t, e, rng))
                for s, t, e in _batch_sizes(case)]
    return _problem(case["kind"], case["dim"], case["side"], case["order"], case["targets"], case["eps"], rng)


def _params(case, eps):
    return SolverParameters(epsilon=eps, tau=TAU if case["kind"] == "trunc" else 0.0, use_log_sum_exp_trick=True,
                            tolerance=1e-8, solver_control_type="linf", verbose_output=False,
                            max_iterations=SOLVE_STEPS if case["kind"] == "solve" else 10000)


def prepare(case, seed):
    if case["kind"] == "batch":
        solver, psis = BatchSolver(case["dim"]), []
        for _, _, eps, (src, y, nu, psi) in _problems(case, seed):
            solver.add_source(src, y, nu, _params(case, eps))
            psis.append(psi)
        return {"case": case, "solver": solver, "psi": psis}
    src, y, nu, psi = _problems(case, seed)
    solver = SotSolver(case["dim"], precision=case["prec"])
    solver.setup_source_measure(src)
    solver.setup_target(y, nu)
    solver.configure(_params(case, case["eps"]))
    state = {"case": case, "solver": solver, "psi": psi}
    if case["kind"] == "solve":
        state["psi"] = np.zeros(case["targets"])
    elif case["host"]:
        state["grad"] = np.empty(case["targets"])
    else:
        n = case["targets"]
        state["psi"] = torch.from_numpy(psi).cuda()
        state["grad"] = torch.empty(n, dtype=torch.float64, device="cuda")
        if case["kind"] == "hessian":
            state["H"] = torch.empty((n, n), dtype=torch.float32, device="cuda")
    return state


def run(state):
    case, solver, psi = state["case"], state["solver"], state["psi"]
    if case["kind"] == "batch":
        values, grads = solver.evaluate(psi, fp32=case["prec"] != "fp64")
        return {"value": values, "grad": np.concatenate(grads)}
    if case["kind"] == "solve":
        return {"psi": solver.solve(psi.copy())}
    if case["kind"] == "hessian":
        solver.compute_hessian_device(psi.data_ptr(), state["H"].data_ptr(), "tensor", out_f32=True)
        return {"H": state["H"]}
    grad = state["grad"]
    if case["host"]:
        value = solver.evaluate_functional(psi, grad)
    else:
        value = solver.evaluate_functional_device(psi.data_ptr(), grad.data_ptr())
    return {"value": np.float64(value), "grad": grad, "C": np.float64(solver.get_C_global())}


# ------------------------------------------------------------------------------------------------------ work

def _points(kind, dim, side, order):
    if kind == "tet":
        return 24 * side ** 3 * {1: 1, 2: 4, 3: 10}[order]
    return (side * order) ** dim


def _eval_work(kind, dim, side, order, targets, eps):
    q = _points(kind, dim, side, order)
    pairs = float(q) * targets
    if kind == "trunc":
        # the ball of the truncation radius at a potential near zero (targets taken as spread evenly)
        r = math.sqrt(max(0.0, 2.0 * eps * math.log(1e-3 / targets / TAU)) + 4.0 * eps)
        pairs *= min(1.0, math.pi * r * r if dim == 2 else 4.0 / 3.0 * math.pi * r ** 3)
    # points, weights and densities; target points, weights and potentials; the gradient
    bytes_ = 8.0 * (q * (dim + 2) + targets * (dim + 2) + targets)
    return bytes_, 4.0 * pairs   # one multiply-add into the point's sum and one into the target's per pair


def work(case):
    dim, order = case["dim"], case["order"]
    if case["kind"] == "batch":
        each = [_eval_work("dense", dim, s, order, t, e) for s, t, e in _batch_sizes(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    b, f = _eval_work(case["kind"], dim, case["side"], order, case["targets"], case["eps"])
    if case["kind"] == "hessian":
        n, q = case["targets"], _points("hessian", dim, case["side"], order)
        return {"bytes": b + 4.0 * n * n, "flops": float(q) * n * n}   # the upper triangle of P^T W P
    if case["kind"] == "solve":
        return {"bytes": b * (SOLVE_STEPS + 1), "flops": f * (SOLVE_STEPS + 1)}
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------- values in 64 bits

def _device(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64).cuda()


def _dense_exact(src, y, nu, psi, eps, probabilities=None):
    """J, its gradient and C over every (point, target) pair, in chunks of points."""
    x, rho, jxw = _device(src["x"]), _device(src["density"]), _device(src["jxw"])
    y, nu, psi = _device(y), _device(nu), _device(psi)
    grad = torch.zeros_like(nu)
    value = torch.zeros((), dtype=torch.float64, device="cuda")
    C = torch.zeros_like(value)
    step = max(1, 100_000_000 // y.shape[0])
    for a in range(0, x.shape[0], step):
        X, w = x[a:a + step], (rho * jxw)[a:a + step]
        d2 = (X[:, :1] - y[:, 0]) ** 2
        for k in range(1, X.shape[1]):
            d2 += (X[:, k:k + 1] - y[:, k]) ** 2
        t = (psi - 0.5 * d2) / eps
        m = t.max(dim=1, keepdim=True).values
        P = nu * torch.exp(t - m)
        S = P.sum(dim=1, keepdim=True)
        value += (w * eps * (m + torch.log(S)).squeeze(1)).sum()
        C += (w / S.squeeze(1)).sum()
        P /= S
        grad += w @ P
        if probabilities is not None:
            probabilities(w, P)
    return value - (psi * nu).sum(), grad - nu, C


def _trunc_exact(src, y, nu, psi, eps):
    """The same over the pairs whose target is within the radius of the point's cell centre."""
    x, w = _device(src["x"]), _device(src["density"] * src["jxw"])
    centres = _device(src["cell_centers"])
    per = x.shape[0] // centres.shape[0]
    radius2 = max(0.0, -2.0 * eps * math.log(TAU / float(nu.min())) + 2.0 * float(psi.max()))
    y, nu, psi = _device(y), _device(nu), _device(psi)
    grad = torch.zeros_like(nu)
    value = torch.zeros((), dtype=torch.float64, device="cuda")
    C = torch.zeros_like(value)
    step = max(1, 60_000_000 // y.shape[0])
    for a in range(0, centres.shape[0], step):
        cc = centres[a:a + step]
        d2 = (cc[:, :1] - y[:, 0]) ** 2
        for k in range(1, cc.shape[1]):
            d2 += (cc[:, k:k + 1] - y[:, k]) ** 2
        cell, j = torch.nonzero(torch.sqrt(d2) <= math.sqrt(radius2), as_tuple=True)
        del d2
        X = x[a * per:(a + cc.shape[0]) * per].view(-1, per, x.shape[1])
        W = w[a * per:(a + cc.shape[0]) * per].view(-1, per)
        t = (psi[j][:, None] - 0.5 * ((X[cell] - y[j][:, None, :]) ** 2).sum(dim=2)) / eps
        m = torch.full_like(W, -math.inf).scatter_reduce(0, cell[:, None].expand_as(t), t, "amax")
        e = nu[j][:, None] * torch.exp(t - m[cell])
        S = torch.zeros_like(W).index_add_(0, cell, e)
        some = S > 0
        value += torch.where(some, W * eps * (m + torch.log(S)), torch.zeros_like(W)).sum()
        C += torch.where(some, W / S, torch.zeros_like(W)).sum()
        grad.index_add_(0, j, (W[cell] * e / S[cell]).sum(dim=1))
    return value - (psi * nu).sum(), grad - nu, C


def exact(case, seed):
    kind, eps = case["kind"], case["eps"]
    if kind == "solve":
        return None
    if kind == "batch":
        got = [_dense_exact(*p, e) for _, _, e, p in _problems(case, seed)]
        return {"value": torch.stack([v for v, _, _ in got]), "grad": torch.cat([g for _, g, _ in got])}
    problem = _problems(case, seed)
    if kind == "hessian":
        n = case["targets"]
        H = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        mass = torch.zeros(n, dtype=torch.float64, device="cuda")

        def add(w, P):
            mass.add_(w @ P)
            H.addmm_((P * w[:, None]).T, P, alpha=-1.0 / eps)

        _dense_exact(*problem, eps, probabilities=add)
        H.diagonal().add_(mass / eps)
        return {"H": H}
    value, grad, C = (_trunc_exact if kind == "trunc" else _dense_exact)(*problem, eps)
    return {"value": value, "grad": grad, "C": C}
