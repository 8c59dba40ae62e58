"""Which sweeps an untruncated evaluation of a structured source takes, and the lattice sweeps (csrc/sdot_lattice.cuh)
where those take them, against the FP64 oracle.

Tolerances as in test_gpu_parity.py: value and C 1e-10 relative, gradient 1e-12 absolute in FP64 and
max(1e-8, 5e-6 max nu_j) where it runs in FP32."""
import numpy as np
import pytest

from semidiscreteot_b200 import BatchSolver, SolverParameters, SotSolver, structured_source

pytestmark = pytest.mark.gpu


def solver_of(src, y, nu, eps, precision):
    s = SotSolver(dim=y.shape[1], device=0, precision=precision)
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    return s


@pytest.mark.parametrize("dim,n,order,N,tiles", [
    (2, 32, 2, 1024, 1), (2, 32, 2, 1025, 0),       # few points: only where all targets are listed
    (2, 48, 2, 3001, 0), (2, 52, 2, 3001, 4), (2, 75, 2, 3001, 9), (2, 64, 3, 1025, 9),
    (3, 8, 2, 1024, 1), (3, 8, 2, 1025, 0), (3, 13, 2, 1025, 0), (3, 14, 2, 1025, 8), (3, 16, 2, 1025, 8),
    (2, 11, 3, 33, 0), (3, 9, 2, 33, 0),            # 33 and 18 points per axis: more padding than points
])
def test_sources_that_take_the_lattice(dim, n, order, N, tiles):
    rng = np.random.default_rng(1)
    s = solver_of(structured_source(dim, n, order), rng.random((N, dim)), np.full(N, 1.0 / N), 1e-2, "fp64")
    assert s.dense_sweeps()["tiles"] == tiles
    s.close()


def tolerance(nu, fp32):
    return max(1e-8, 5e-6 * float(np.max(nu))) if fp32 else 1e-12


def oracle_of(orc, src, y, nu, eps, psi, lse=True):
    P = orc.Problem(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"], y, nu)
    return P.evaluate(psi, orc.Params(epsilon=eps, tau=0.0, use_log_sum_exp=lse))


def graded(dim, n, order, seed=3):
    """A lattice without a period: every dimension stretched by the same smooth map (cells of different widths)."""
    src = dict(structured_source(dim, n, order, nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0])))
    stretch = lambda t: t + 0.1 * np.sin(np.pi * t) ** 2
    src["x"], src["cell_centers"] = stretch(src["x"]), stretch(src["cell_centers"])
    return src


# (dim, cells per axis, order, targets, eps, tile, tiles, runs)
LATTICE = [
    (2, 32, 2, 1, 2e-2, 64, 1, 1),        # one full tile; one target, fewer than a fragment, one more than a chunk
    (2, 32, 2, 5, 2e-2, 64, 1, 1),
    (2, 22, 3, 33, 1e-2, 64, 4, 1),       # 66 points: second tiles of 2
    (2, 43, 3, 700, 1e-2, 64, 9, 1),      # 129 points: third tiles of 1
    (2, 16, 4, 65, 1e-2, 64, 1, 1),       # a period of 4 points
    (2, 60, 1, 40, 1e-2, 64, 1, 1),       # a period of 1 point, 60 of them
    (2, 10, 3, 130, 1e-2, 64, 1, 1),      # 30 points: half a tile
    (2, 56, 2, 1025, 1e-2, 64, 4, 1),     # more targets than are listed: the target blocks
    (2, 65, 3, 3000, 5e-3, 64, 16, 1),    # 195 points: fourth tiles of 3
    (2, 56, 2, 1100, 9e-4, 32, 16, 1),    # tiles of 32 (and 16) points
    (2, 64, 2, 1500, 1.2e-3, 64, 4, 1),   # factors of 300 bits
    (3, 8, 2, 64, 1e-2, 16, 1, 1),        # one full tile, one full block of targets
    (3, 7, 2, 9, 1e-2, 16, 1, 1),         # 14 points
    (3, 14, 2, 1300, 1e-2, 16, 8, 1),     # 28 points: second tiles of 12; target blocks
    (3, 18, 2, 1025, 1e-2, 16, 27, 1),    # 36 points: third tiles of 4
    (3, 10, 3, 1100, 2e-2, 16, 8, 1),     # 27-point cells: a period of 3
    (3, 10, 3, 65, 4e-3, 16, 8, 1),
    (3, 10, 3, 65, 1.65e-3, 16, 8, 0),    # a run covers a tile, whose factors span 330 bits: one exponential each
]


@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("dim,n,order,N,eps,tile,tiles,runs", LATTICE)
def test_lattice_sweeps(oracle_mod, dim, n, order, N, eps, tile, tiles, runs, precision):
    rng = np.random.default_rng(100 * n + N)
    src = structured_source(dim, n, order, nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0]))
    y, nu = rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5)
    s = solver_of(src, y, nu, eps, precision)
    sweeps = s.dense_sweeps()
    assert (sweeps["tile"], sweeps["tiles"], sweeps["runs"]) == (tile, tiles, runs)
    assert sweeps["lattice_gradient"] == (precision == "fp64")
    for k in range(3):  # eager, eager or captured, replayed
        psi, g = 0.5 * eps * rng.standard_normal(N), np.zeros(N)
        J = s.evaluate_functional(psi, g)
        J0, g0, st = oracle_of(oracle_mod, src, y, nu, eps, psi)
        assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6), (k, J, J0)
        tol = tolerance(nu, precision != "fp64")
        if precision != "fp64" and eps < 5e-3:  # FP32 exponents of up to dim / (2 eps), rounded four times
            tol = max(tol, 4 * 2.0 ** -24 * dim / (2 * eps) * float(np.max(g0 + nu)))
        assert np.max(np.abs(g - g0)) <= tol, (k, np.max(np.abs(g - g0)))
        assert abs(s.get_C_global() - st["C_global"]) <= 1e-10 * abs(st["C_global"]), k
    s.close()


@pytest.mark.parametrize("lse", [True, False])
@pytest.mark.parametrize("dim,n,order,N,tiles", [(2, 23, 3, 500, 4), (2, 40, 3, 1200, 4), (3, 8, 2, 300, 1), (3, 14, 2, 1100, 8)])
def test_lattice_without_a_period(oracle_mod, dim, n, order, N, tiles, lse):
    rng = np.random.default_rng(n)
    src, eps = graded(dim, n, order), 2e-2
    y, nu, psi, g = rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5), 0.5 * eps * rng.standard_normal(N), np.zeros(N)
    s = solver_of(src, y, nu, eps, "fp64")
    s.configure(SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=lse))
    sweeps = s.dense_sweeps()
    assert (sweeps["tiles"], sweeps["runs"]) == (tiles, 0)
    J = s.evaluate_functional(psi, g)
    J0, g0, st = oracle_of(oracle_mod, src, y, nu, eps, psi, lse)
    assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6)
    assert np.max(np.abs(g - g0)) <= 1e-12
    assert abs(s.get_C_global() - st["C_global"]) <= 1e-10 * abs(st["C_global"])
    s.close()


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_batched_lattices(oracle_mod, dim, fp32):
    """Listed targets and target blocks (members in k-d order), ragged tiles, several slices, no period, and problems
    that are no lattice between them."""
    rng = np.random.default_rng(dim)
    sizes = ([(32, 2, 1100, 5e-3, 1), (10, 3, 130, 1e-2, 1), (50, 3, 1500, 1e-2, 1), (9, 2, 65, 2e-2, 0), (43, 3, 33, 5e-3, 1)]
             if dim == 2 else [(8, 2, 1100, 1e-2, 1), (14, 2, 300, 1e-2, 1), (5, 2, 65, 2e-2, 0), (13, 3, 1030, 1e-2, 1)])
    probs = []
    b = BatchSolver(dim=dim)
    for k, (n, order, N, eps, _) in enumerate(sizes):
        src = graded(dim, n, order) if k == 1 else structured_source(dim, n, order)
        y, nu = rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5)
        b.add_source(src, y, nu, SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
        probs.append((src, y, nu, eps, 0.5 * eps * rng.standard_normal(N)))
    vals, grads = b.evaluate([p[4] for p in probs], fp32=fp32)
    for k, ((src, y, nu, eps, psi), J, g) in enumerate(zip(probs, vals, grads)):
        sweeps = b.sweeps(k)
        assert (sweeps["tile"] > 0) == bool(sizes[k][4]) and sweeps["lattice_gradient"] == (sweeps["tile"] > 0 and not fp32)
        J0, g0, _ = oracle_of(oracle_mod, src, y, nu, eps, psi)
        assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6)
        assert np.max(np.abs(g - g0)) <= tolerance(nu, fp32)
    b.close()
