"""Untruncated sweeps over tensor lattices of points (csrc/sdot_lattice.cuh) against the FP64 oracle, at the edges
of their tiles: 64 x 64 or 16 x 16 x 16 points (32 x 32 where the factors of a tile would leave the FP64 range),
chunks of 32 targets, blocks of 64 targets, 1,024 listed targets, runs of 8 points a period apart.

Tolerances as in test_gpu_parity.py: value and C 1e-10 relative, gradient 1e-12 absolute in FP64 and
max(1e-8, 5e-6 max nu_j) in the hybrid mode."""
import numpy as np
import pytest

from cell_sources import graded_source
from semidiscreteot_b200 import SolverParameters, SotSolver, structured_source

pytestmark = pytest.mark.gpu

# (dim, cells per axis, order, targets, epsilon)
CASES = [
    (2, 32, 2, 1024, 2e-2),   # one full tile, the last size whose targets are all listed
    (2, 11, 3, 1025, 1e-2),   # 33 points: past half a tile; the first size that goes by target blocks
    (2, 22, 3, 33, 1e-2),     # 66 points: a second tile of 2; a second chunk of 1 target
    (2, 43, 3, 1500, 2e-3),   # 129 points: three tiles, the last of 1
    (2, 16, 3, 700, 1e-3),    # factors of a 48-point tile too far apart: tiles of 32 and 16
    (2, 7, 1, 5, 1e-1),       # one point per cell, fewer targets than a fragment
    (2, 40, 1, 1, 5e-2),      # one target
    (3, 8, 2, 64, 1e-2),      # one full tile, one full block of targets
    (3, 9, 2, 1300, 5e-3),    # 18 points: second tiles of 2 in every dimension
    (3, 6, 3, 65, 1e-2),      # 27-point cells (no cell sweep exists for these)
    (3, 5, 2, 40, 5e-4),      # outside the FP64 range of the factors: the cell sweeps
]


def check(orc, src, y, nu, eps, precision, seed):
    rng = np.random.default_rng(seed)
    dim = y.shape[1]
    s = SotSolver(dim=dim, device=0, precision=precision)
    s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
    s.setup_target(y, nu)
    s.configure(SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    P = orc.Problem(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"], y, nu)
    op = orc.Params(epsilon=eps, tau=0.0, use_log_sum_exp=True)
    tol = 1e-12 if precision == "fp64" else max(1e-8, 5e-6 * float(np.max(nu)))
    for k in range(3):  # eager, eager or captured, replayed
        psi = 0.5 * eps * rng.standard_normal(len(nu))
        g = np.zeros(len(nu))
        J = s.evaluate_functional(psi, g)
        Jo, go, st = P.evaluate(psi, op)
        assert abs(J - Jo) <= 1e-10 * max(abs(Jo), 1e-6), (k, J, Jo)
        assert np.max(np.abs(g - go)) <= tol, (k, np.max(np.abs(g - go)))
        assert abs(s.get_C_global() - st["C_global"]) <= 1e-10 * abs(st["C_global"]), k
    s.close()


# The last case's gradient runs on the cell sweep, whose FP32 form is 2.4e-7 off there against its bound of
# 2.1e-7: the bound does not hold at 40 targets and eps = 5e-4.
FP32_GRADIENT = pytest.mark.xfail(strict=True, reason="FP32 cell sweep beyond its gradient bound at eps = 5e-4")


@pytest.mark.parametrize("case,precision", [
    pytest.param(c, p, id="%dd_%dx%d_%d-%s" % (*c[:4], p),
                 marks=[FP32_GRADIENT] if c == CASES[-1] and p == "hybrid" else [])
    for c in CASES for p in ("fp64", "hybrid")])
def test_lattice_tile_edges(oracle_mod, case, precision):
    dim, n, order, N, eps = case
    rng = np.random.default_rng(100 * n + N)
    src = structured_source(dim, n, order, nodal_density=lambda p: 1.0 + 0.5 * np.sin(3.0 * p[:, 0]))
    check(oracle_mod, src, rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5), eps, precision, n)


@pytest.mark.parametrize("kind", ["graded", "moved", "missing", "shuffled"])
def test_lattices_without_period_and_no_lattices(oracle_mod, kind):
    """Coordinates without a period (one exponential per factor); one point moved and one cell missing (no
    lattice: the cell or point sweeps); the cells in another order (the same lattice)."""
    rng = np.random.default_rng(8)
    src = graded_source(rng, 2, 23, 3) if kind == "graded" else structured_source(2, 23, 3)
    x, ncell = src["x"].reshape(-1, 9, 2).copy(), src["cell_centers"].shape[0]
    keep = np.arange(ncell)
    if kind == "moved":
        x[5, 4] += 1e-4
    elif kind == "missing":
        keep = np.delete(keep, 100)
    elif kind == "shuffled":
        keep = rng.permutation(ncell)
    per_cell = lambda a: a.reshape(ncell, 9)[keep].ravel()
    src = dict(x=x[keep].reshape(-1, 2), jxw=per_cell(src["jxw"]), density=per_cell(src["density"]),
               cell_offsets=np.arange(len(keep) + 1) * 9, cell_centers=src["cell_centers"][keep])
    N = 500
    check(oracle_mod, src, rng.random((N, 2)), np.full(N, 1.0 / N), 1e-2, "fp64", 3)


def test_another_source_of_the_same_size():
    """A second source of the same size on one solver (same buffers, other lattice): the captured graph of the
    first is not replayed for it."""
    rng = np.random.default_rng(4)
    N, eps = 300, 2e-2
    y, nu = rng.random((N, 2)), np.full(N, 1.0 / N)
    psi = 0.3 * eps * rng.standard_normal(N)
    prm = SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True)

    def setup(s, src):
        s.setup_source(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"])
        s.setup_target(y, nu)
        s.configure(prm)

    def evaluate(s):
        g = np.zeros(N)
        return s.evaluate_functional(psi, g), g

    a = structured_source(2, 12, 3)
    b = graded_source(rng, 2, 12, 3)
    one = SotSolver(dim=2, device=0, precision="fp64")
    setup(one, a)
    for _ in range(4):
        Ja, ga = evaluate(one)
    setup(one, b)
    Jb, gb = evaluate(one)
    fresh = SotSolver(dim=2, device=0, precision="fp64")
    setup(fresh, b)
    Jf, gf = evaluate(fresh)
    assert Jb == Jf and np.array_equal(gb, gf)
    assert Ja != Jb
    one.close()
    fresh.close()
