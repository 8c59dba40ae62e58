"""Which sweeps an untruncated evaluation of a structured source takes, and the lattice sweeps (csrc/sdot_lattice.cuh)
where those take them, against the FP64 oracle.

Tolerances as in test_gpu_parity.py: value and C 1e-10 relative, gradient 1e-12 absolute in FP64 and
max(1e-8, 5e-6 max nu_j) where it runs in FP32."""
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


@pytest.mark.parametrize("dim,n,order,N,tiles", [
    (2, 32, 2, 1024, 1), (2, 32, 2, 1025, 0),       # few points: only where all targets are listed
    (2, 52, 2, 3001, 0), (2, 56, 2, 3001, 4), (2, 75, 2, 3001, 9), (2, 64, 3, 1025, 9),
    (3, 8, 2, 1024, 1), (3, 8, 2, 1025, 0), (3, 13, 2, 1025, 0), (3, 14, 2, 1025, 8), (3, 16, 2, 1025, 8),
    (2, 11, 3, 33, 0), (3, 9, 2, 33, 0),            # 33 and 18 points per axis: more padding than points
])
def test_sources_that_take_the_lattice(dim, n, order, N, tiles):
    rng = np.random.default_rng(1)
    s = solver_of(structured_source(dim, n, order), rng.random((N, dim)), np.full(N, 1.0 / N), 1e-2, "fp64")
    assert s.dense_sweeps()["tiles"] == tiles
    s.close()
