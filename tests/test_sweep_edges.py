"""Sweeps over sources without grid structure, the truncated sweeps' lists and chunks, batches of mixed sources and
the covering radius, at the sizes where their tiles end, against the FP64 oracle.

Tolerances as in test_gpu_parity.py: value and C 1e-10 relative, gradient 1e-12 absolute in FP64 and
max(1e-8, 5e-6 max nu_j) where it runs in FP32; pair counts and covering radii equal."""
import numpy as np
import pytest

from semidiscreteot_b200 import BatchSolver, SolverParameters, SotSolver, structured_source

pytestmark = pytest.mark.gpu


def jittered(dim, n, order, seed):
    """A structured source with every point moved a little: no lattice, no tensor cells."""
    src = dict(structured_source(dim, n, order, nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0])))
    src["x"] = src["x"] + 0.1 / n * np.random.default_rng(seed).uniform(-1, 1, src["x"].shape)
    return src


def oracle_of(orc, src, y, nu):
    return orc.Problem(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"], y, nu)


def check(orc, src, y, nu, eps, tau, precision, psis):
    s = SotSolver(dim=y.shape[1], device=0, precision=precision)
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=tau, use_log_sum_exp_trick=True))
    P = oracle_of(orc, src, y, nu)
    tol = 1e-12 if precision == "fp64" else max(1e-8, 5e-6 * float(np.max(nu)))
    for psi in psis:
        g = np.zeros(len(nu))
        J = s.evaluate_functional(psi, g)
        Jo, go, st = P.evaluate(psi, orc.Params(epsilon=eps, tau=tau, use_log_sum_exp=True))
        if tau > 0:
            assert s.last_eval_info["n_pairs"] == st["n_pairs"]
        assert abs(J - Jo) <= 1e-10 * max(abs(Jo), 1e-6), (J, Jo)
        assert np.max(np.abs(g - go)) <= tol, np.max(np.abs(g - go))
        assert abs(s.get_C_global() - st["C_global"]) <= 1e-10 * abs(st["C_global"])
    s.close()


# (dim, cells per axis, order, targets): steps of 8 targets, 256 staged at a time, 128 points per block, octets of
# points of four groups, one block of points per SM slot (no target slices) or fewer
@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("dim,n,order,N", [(2, 3, 3, 1), (2, 8, 2, 7), (2, 9, 3, 8), (2, 37, 2, 257), (3, 4, 2, 9),
                                           (3, 5, 3, 1025), (2, 92, 3, 264), (3, 22, 2, 250)])
def test_point_sweeps(oracle_mod, dim, n, order, N, precision):
    rng = np.random.default_rng(N)
    eps = 2e-2
    check(oracle_mod, jittered(dim, n, order, n), rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5), eps, 0.0,
          precision, [0.5 * eps * rng.standard_normal(N) for _ in range(2)])


@pytest.mark.parametrize("order", ["rising", "falling", "random"])
def test_point_sweep_reference_moves(oracle_mod, order):
    """Potentials that differ by 800 eps: the reference of the sums moves (rising) or the early targets' exponent
    stays the largest (falling)."""
    rng = np.random.default_rng(4)
    N, eps = 500, 1e-2
    psi = 800 * eps * np.linspace(0, 1, N)
    psi = psi[::-1].copy() if order == "falling" else (rng.permutation(psi) if order == "random" else psi)
    check(oracle_mod, jittered(3, 6, 2, 1), rng.random((N, 3)), rng.dirichlet(np.ones(N) * 5), eps, 0.0, "fp64", [psi])


@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("dim,n,order", [(2, 24, 2), (2, 24, 3), (3, 8, 2), (3, 7, 2), (2, 12, 4)])
def test_truncated_lists_and_chunks(oracle_mod, dim, n, order, precision):
    """A tight cluster (several chunks per source block) around 300 targets that nearly coincide (more candidates for
    a point's largest exponent than its list holds), and a few targets far away; in 3D, source blocks of 2 x 2 x 2
    cells and ragged ones."""
    rng = np.random.default_rng(dim * n + order)
    y = np.concatenate([0.5 + 0.02 * rng.standard_normal((2500, dim)), 0.45 + 1e-7 * rng.standard_normal((300, dim)),
                        rng.random((101, dim))])
    y = np.clip(y, 0, 1)
    nu = rng.dirichlet(np.ones(len(y)) * 2)
    check(oracle_mod, structured_source(dim, n, order), y, nu, 2e-3, 1e-10, precision,
          [1e-3 * rng.standard_normal(len(y))])


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_batch_of_mixed_sources(oracle_mod, dim, fp32):
    rng = np.random.default_rng(dim)
    b = BatchSolver(dim=dim)
    probs = []
    for n, order, N, grid in [(9, 2, 65, True), (5, 3, 1, False), (12, 2, 700, False), (4, 1, 33, True)]:
        src = structured_source(dim, n, order) if grid else jittered(dim, n, order, n)
        y, nu = rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5)
        b.add_source(src, y, nu, SolverParameters(epsilon=2e-2, tau=0.0, use_log_sum_exp_trick=True))
        probs.append((src, y, nu, 1e-2 * rng.standard_normal(N)))
    vals, grads = b.evaluate([p[3] for p in probs], fp32=fp32)
    for (src, y, nu, psi), J, g in zip(probs, vals, grads):
        Jo, go, _ = oracle_of(oracle_mod, src, y, nu).evaluate(
            psi, oracle_mod.Params(epsilon=2e-2, tau=0.0, use_log_sum_exp=True))
        assert abs(J - Jo) <= 1e-10 * max(abs(Jo), 1e-6)
        assert np.max(np.abs(g - go)) <= (max(1e-8, 5e-6 * nu.max()) if fp32 else 1e-12)
    b.close()


@pytest.mark.parametrize("dim,n,N", [(2, 3, 1), (2, 30, 700), (3, 7, 33), (3, 30, 3000)])
def test_covering_radius(oracle_mod, dim, n, N):
    """Few cells (several threads share one) and many, against the oracle's radius."""
    rng = np.random.default_rng(n)
    src, y, nu = structured_source(dim, n, 2), rng.random((N, dim)), np.full(N, 1.0 / N)
    s = SotSolver(dim=dim, device=0, precision="fp64")
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    assert s.compute_covering_radius() == oracle_of(oracle_mod, src, y, nu).covering_radius()
    s.close()


@pytest.mark.parametrize("dim,n,order,N,eps", [(2, 16, 3, 200, 1e-3), (2, 12, 3, 100, 4e-4), (2, 48, 2, 800, 3e-4),
                                               (3, 12, 2, 600, 2e-3), (3, 16, 2, 1500, 5e-4)])
def test_truncated_fp64_gradient_relative(oracle_mod, dim, n, order, N, eps):
    """FP64 gradient over tensor-product points, per target relative to its mass: exponents of up to 40 (natural
    units) rounded eight times each here and in the oracle, 2 x 8 x 40 x 2^-53 = 7.1e-14, and nothing from the
    exponentials, whose products are good to a few ulp."""
    rng = np.random.default_rng(n + N)
    src = structured_source(dim, n, order, nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0]))
    y, nu = rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5)
    psi, g = 0.5 * eps * rng.standard_normal(N), np.zeros(N)
    s = SotSolver(dim=dim, device=0, precision="fp64")
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=1e-12, use_log_sum_exp_trick=True))
    s.evaluate_functional(psi, g)
    s.close()
    _, g0, _ = oracle_of(oracle_mod, src, y, nu).evaluate(
        psi, oracle_mod.Params(epsilon=eps, tau=1e-12, use_log_sum_exp=True))
    mass = g0 + nu
    assert np.max((np.abs(g - g0) / mass)[mass > 1e-8]) <= 2 * 8 * 40 * 2.0 ** -53
