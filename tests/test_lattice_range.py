"""The ends of the range of the lattice sweeps (csrc/sdot_lattice.cuh) against the FP64 oracle: elongated sources,
whose factors span the whole admitted range along one axis, and sources away from the origin, whose coordinates are
rounded.

Tolerances as in test_gpu_parity.py: value and C 1e-10 relative, gradient 1e-12 absolute in FP64. Where it runs in
FP32, the exponent's terms of up to D^2 / (2 eps) (D: the largest distance) are rounded four times: a relative
error of 4 2^-24 D^2 / (2 eps) of a target's mass, which exceeds max(1e-8, 5e-6 max nu_j) at the eps used here."""
import numpy as np
import pytest

from semidiscreteot_b200 import BatchSolver, SolverParameters, SotSolver, structured_source

pytestmark = pytest.mark.gpu


def box_source(cells, order, size):
    """Gauss points of a uniform mesh of `cells` hexahedra (or quadrilaterals) on the box of side lengths `size`."""
    dim = len(cells)
    one = structured_source(2, 1, order)               # nodes and weights of one cell, x fastest
    g, w = one["x"][:order, 0], one["jxw"].reshape(order, order).sum(0)
    h = np.asarray(size) / np.asarray(cells)
    corner = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1)
    corner = corner.transpose(*range(dim)[::-1], dim).reshape(-1, dim)
    node = np.stack(np.meshgrid(*[g] * dim, indexing="ij"), -1).transpose(*range(dim)[::-1], dim).reshape(-1, dim)
    weight = np.prod(np.stack(np.meshgrid(*[w] * dim, indexing="ij"), -1), -1).transpose(*range(dim)[::-1]).ravel()
    n, qpc = len(corner), len(node)
    x = (corner[:, None, :] + node[None, :, :]) * h
    return dict(x=x.reshape(-1, dim), jxw=np.tile(weight, n) * np.prod(h), density=np.ones(n * qpc) / np.prod(size),
                cell_offsets=np.arange(n + 1) * qpc, cell_centers=(corner + 0.5) * h)


def tolerance(src, y, nu, eps, want, fp32):
    if not fp32:
        return 1e-12
    lo, hi = (f(np.concatenate([src["x"], y]), axis=0) for f in (np.min, np.max))
    mass = float(np.max(want[1] + nu))
    return max(1e-8, 5e-6 * float(np.max(nu)), 4 * 2.0 ** -24 * np.sum((hi - lo) ** 2) / (2 * eps) * mass)


def solver_of(src, y, nu, eps, precision):
    s = SotSolver(dim=y.shape[1], device=0, precision=precision)
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    return s


def oracle_of(orc, src, y, nu, eps, psi):
    P = orc.Problem(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"], y, nu)
    return P.evaluate(psi, orc.Params(epsilon=eps, tau=0.0, use_log_sum_exp=True))


def check(s, want, psi, tol):
    J0, g0, st = want
    g = np.zeros(len(psi))
    J = s.evaluate_functional(psi, g)
    assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6), (J, J0)
    assert np.max(np.abs(g - g0)) <= tol, np.max(np.abs(g - g0))
    assert abs(s.get_C_global() - st["C_global"]) <= 1e-10 * abs(st["C_global"])


def beam(order=3, axis=0):
    """16 x 4 x 4 cells on 1 x 0.02 x 0.02 and targets at the two ends: with a period of 3 points one run of
    factors covers a tile of 16 points.  axis: the dimension that the beam lies along."""
    rng = np.random.default_rng(5)
    y = rng.random((40, 3)) * [0.02, 0.02, 0.02]
    y[20:, 0] += 0.98
    src = box_source((48 // order, 4, 4), order, (1.0, 0.02, 0.02))
    turn = lambda a: np.ascontiguousarray(np.roll(a, axis, axis=1))
    src["x"], src["cell_centers"] = turn(src["x"]), turn(src["cell_centers"])
    return src, turn(y), rng.dirichlet(np.ones(40) * 5)


BEAM_EPS = [3.2e-4, 3.25e-4, 3.3e-4, 3.4e-4, 3.45e-4, 3.6e-4, 4e-4, 4.5e-4, 4.8e-4, 5e-4, 5.2e-4, 5.5e-4, 6e-4]


@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("eps", BEAM_EPS)
def test_beam(oracle_mod, order, eps, precision):
    src, y, nu = beam(order)
    s = solver_of(src, y, nu, eps, precision)
    psi = np.zeros(len(nu))
    want = oracle_of(oracle_mod, src, y, nu, eps, psi)
    check(s, want, psi, tolerance(src, y, nu, eps, want, precision != "fp64"))
    s.close()


@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("eps", BEAM_EPS)
def test_beam_along_another_axis(oracle_mod, axis, eps):
    src, y, nu = beam(3, axis)
    s = solver_of(src, y, nu, eps, "fp64")
    psi = np.zeros(len(nu))
    check(s, oracle_of(oracle_mod, src, y, nu, eps, psi), psi, 1e-12)
    s.close()


@pytest.mark.parametrize("fp32", [False, True])
def test_beams_in_a_batch(oracle_mod, fp32):
    b = BatchSolver(dim=3)
    probs = [beam(order) + (eps,) for order in (2, 3) for eps in BEAM_EPS[::2]]
    for src, y, nu, eps in probs:
        b.add_source(src, y, nu, SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    psis = [np.zeros(len(p[2])) for p in probs]
    vals, grads = b.evaluate(psis, fp32=fp32)
    for (src, y, nu, eps), psi, J, g in zip(probs, psis, vals, grads):
        want = oracle_of(oracle_mod, src, y, nu, eps, psi)
        J0, g0, _ = want
        assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6), (eps, J, J0)
        assert np.max(np.abs(g - g0)) <= tolerance(src, y, nu, eps, want, fp32), (eps, np.max(np.abs(g - g0)))
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("offset", [-300.0, 1e3, 1e5])
@pytest.mark.parametrize("dim,n,order,N,eps", [(2, 64, 2, 400, 1.7e-3), (2, 43, 3, 400, 1.7e-3), (3, 8, 2, 64, 5e-3)])
def test_source_away_from_the_origin(oracle_mod, dim, n, order, N, eps, offset, precision):
    """The unit cube moved by `offset`: its coordinates are rounded to ulps of the offset, which neither equal
    steps nor merged coordinates may add to the exponents (those are formed about the source's centre)."""
    rng = np.random.default_rng(n)
    src = structured_source(dim, n, order, lo=offset, hi=offset + 1.0,
                            nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0]))
    y, nu = offset + rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5)
    psi = 0.5 * eps * rng.standard_normal(N)
    s = solver_of(src, y, nu, eps, precision)
    want = oracle_of(oracle_mod, src, y, nu, eps, psi)
    check(s, want, psi, tolerance(src, y, nu, eps, want, precision != "fp64"))
    s.close()


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e4])
def test_coordinates_rounded_cell_by_cell(oracle_mod, scale):
    """Points whose shared coordinates differ in the last bits (each cell mapped by itself)."""
    rng = np.random.default_rng(2)
    src = dict(structured_source(2, 64, 2))
    src["x"] = src["x"] + 2.0 ** -53 * rng.integers(-1, 2, src["x"].shape)
    src["x"], src["cell_centers"] = scale * src["x"], scale * src["cell_centers"]
    N, eps = 400, 1.7e-3 * scale ** 2
    y, nu, psi = scale * rng.random((N, 2)), rng.dirichlet(np.ones(N) * 5), 0.5 * eps * rng.standard_normal(N)
    s = solver_of(src, y, nu, eps, "fp64")
    check(s, oracle_of(oracle_mod, src, y, nu, eps, psi), psi, 1e-12)
    s.close()
