"""Batched evaluations of problems on tensor lattices: their memory, and what a problem's results depend on."""
import numpy as np
import pytest

from semidiscreteot_b200 import BatchSolver, SolverParameters, _lib, structured_source

pytestmark = pytest.mark.gpu


def problem(dim, n, order, N, eps=2e-2, seed=0):
    rng = np.random.default_rng([seed, n, N])
    return (structured_source(dim, n, order), rng.random((N, dim)), rng.dirichlet(np.ones(N) * 5), eps,
            0.5 * eps * rng.standard_normal(N))


def batch_of(dim, probs):
    b = BatchSolver(dim=dim)
    for src, y, nu, eps, _ in probs:
        b.add_source(src, y, nu, SolverParameters(epsilon=eps, tau=0.0, use_log_sum_exp_trick=True))
    return b


def check(orc, probs, vals, grads):
    for (src, y, nu, eps, psi), J, g in zip(probs, vals, grads):
        P = orc.Problem(src["x"], src["jxw"], src["density"], src["cell_offsets"], src["cell_centers"], y, nu)
        J0, g0, _ = P.evaluate(psi, orc.Params(epsilon=eps, tau=0.0, use_log_sum_exp=True))
        assert abs(J - J0) <= 1e-10 * max(abs(J0), 1e-6)
        assert np.max(np.abs(g - g0)) <= 1e-12


PROBLEMS = [(2, 16, 3, 300), (2, 10, 3, 130), (2, 32, 2, 1100), (2, 40, 2, 257), (2, 9, 2, 65)]


def test_no_memory_for_the_lattice(oracle_mod):
    """The batch runs without the lattices' buffer (an upload's second) and reports a failure of any other
    allocation."""
    L = _lib.load()
    probs = [problem(*p) for p in PROBLEMS]
    psis = [p[4] for p in probs]
    try:
        for k in range(4):
            b = batch_of(2, probs)
            L.sdot_debug_fail_allocation(k)
            if k == 1:
                vals, grads = b.evaluate(psis)
                L.sdot_debug_fail_allocation(-1)
                assert all(b.sweeps(i)["tile"] == 0 for i in range(len(probs)))
                check(oracle_mod, probs, vals, grads)
                vals2, grads2 = b.evaluate(psis)
                assert np.array_equal(vals, vals2) and all(map(np.array_equal, grads, grads2))
            else:
                with pytest.raises(_lib.SdotError) as e:
                    b.evaluate(psis)
                L.sdot_debug_fail_allocation(-1)
                assert e.value.status == _lib.SDOT_ENOMEM
                check(oracle_mod, probs, *b.evaluate(psis))
            b.close()
    finally:
        L.sdot_debug_fail_allocation(-1)


@pytest.mark.parametrize("cap", [1, 600_000, 1_000_000])
@pytest.mark.parametrize("fp32", [False, True])
def test_groups_of_problems(oracle_mod, monkeypatch, fp32, cap):
    """Slice sums held for a few problems at a time: the bits of all together."""
    probs = [problem(*p) for p in PROBLEMS]
    psis = [p[4] for p in probs]
    b = batch_of(2, probs)
    want = b.evaluate(psis, fp32=fp32)
    assert [b.sweeps(i)["tile"] > 0 for i in range(len(probs))] == [True, True, True, True, False]
    b.close()
    monkeypatch.setenv("SDOT_BATCH_SUMS_BYTES", str(cap))
    b = batch_of(2, probs)
    for _ in range(2):
        vals, grads = b.evaluate(psis, fp32=fp32)
        assert np.array_equal(vals, want[0]) and all(map(np.array_equal, grads, want[1]))
    if not fp32:
        check(oracle_mod, probs, vals, grads)
    b.close()


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("dim,n,order,N", [(2, 32, 2, 3000), (2, 16, 3, 700), (3, 8, 2, 2000), (2, 9, 2, 600)])
def test_results_do_not_depend_on_the_companions(dim, n, order, N, fp32):
    """One problem (on the lattice, and on the point sweeps) alone and in a batch with larger ones."""
    one = problem(dim, n, order, N)
    big = [problem(2, 128, 3, 16384), problem(2, 100, 3, 16000)] if dim == 2 else [problem(3, 32, 2, 20000)]
    out = []
    for probs in ([one], [one] + big, big + [one, problem(dim, n, order, 130)]):
        b = batch_of(dim, probs)
        vals, grads = b.evaluate([p[4] for p in probs], fp32=fp32)
        k = [p is one for p in probs].index(True)
        out.append((vals[k], grads[k]))
        b.close()
    for J, g in out[1:]:
        assert J == out[0][0] and np.array_equal(g, out[0][1])
