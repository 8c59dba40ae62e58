"""sdot_evaluate_device_noalloc against sdot_evaluate_device bit for bit, over the sweeps and scratch sizes that an
untruncated evaluation can take (test_zz_no_alloc.py holds the entry point's other properties)."""
import numpy as np
import pytest

from semidiscreteot_b200 import SolverParameters, SotSolver, structured_source

pytestmark = pytest.mark.gpu


def solver_of(src, y, nu, eps, precision):
    s = SotSolver(dim=y.shape[1], device=0, precision=precision)
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    return s


def problem(dim, n, order, N, seed=1):
    rng = np.random.default_rng(seed)
    return structured_source(dim, n, order), rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5), rng.standard_normal(N)


def both(s, psi):
    """(J, gradient, C) of the allocating and of the no-allocation entry point."""
    import torch
    p = torch.tensor(psi, dtype=torch.float64, device="cuda")
    out = []
    for call in (s.evaluate_functional_device, s.evaluate_functional_device_noalloc):
        g = torch.full_like(p, np.nan)
        J = call(p.data_ptr(), g.data_ptr())
        torch.cuda.synchronize()
        out.append((J, g.cpu().numpy(), s.get_C_global()))
    return out


def assert_same(s, psi):
    (Ja, ga, Ca), (Jn, gn, Cn) = both(s, psi)
    assert Ja == Jn and Ca == Cn and np.array_equal(ga, gn)


def test_calls_of_different_grids_in_turn():
    """Contexts whose finalize grids differ share the scratch and its arrival counter."""
    sizes = [(2, 4, 2, 5), (2, 8, 3, 900), (3, 6, 2, 257), (2, 5, 2, 33)]
    probs = [problem(*c) for c in sizes]
    solvers = [solver_of(src, y, nu, 2e-2, "fp64") for src, y, nu, _ in probs]
    for _ in range(2):
        for s, p in zip(solvers, probs):
            assert_same(s, 1e-2 * p[3])
    for s in solvers:
        s.close()


# lattice partials beyond the scratch (63 or 64 slices x 4 tiles, 37 x 8), those of the cell or point sweeps within it
@pytest.mark.parametrize("precision", ["fp64", "hybrid"])
@pytest.mark.parametrize("dim,n,order,N", [(2, 64, 2, 1024), (2, 64, 2, 1100), (2, 32, 4, 1000),
                                              (3, 8, 4, 1000)])
def test_slices_in_passes(dim, n, order, N, precision):
    src, y, nu, z = problem(dim, n, order, N)
    s = solver_of(src, y, nu, 2e-2, precision)
    for k in range(2):
        assert_same(s, 1e-2 * (k + 1) * z)
    s.close()
