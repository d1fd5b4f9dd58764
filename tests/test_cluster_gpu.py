"""Cluster-resident chunks: a small single LP runs its iterations inside
thread-block clusters, in launches of at most 32 (the default) or of a check
period each (options.cluster_chunks=1), instead of two launches per iteration.

The cluster kernel sums every row in rows_kernel's order and takes the same
steps, so the tests hold both forms to bit-identical iterates, iteration and
restart counts against use_graphs=0, which runs two plain launches per
iteration, in FP32 and FP64:
- the 1000 x 1500 random LP and a refinery case, fixed budgets and whole
  solves with polishing (whose single-case sub-solves take the cluster too);
- an LP with rows of 700 nonzeros (the warp-summed rows);
- an LP with rows longer than 1,024 (not taken: two launches per iteration);
- a case stack, whose last FP32 case is handed to the single-LP path.
The FP64 iterates also match the oracle to 1e-10 after fixed budgets.
"""
import numpy as np
import pytest

import oracle
from anukulan_b200 import lpgen
from anukulan_b200.abi import ITERATION_LIMIT, OPTIMAL, PRECISION_FP32

pytestmark = pytest.mark.gpu

PRECISIONS = [0, PRECISION_FP32]


def same(a, b):
    return (a.status == b.status and a.iterations == b.iterations
            and a.restarts == b.restarts and a.polish_attempts == b.polish_attempts
            and np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y))


def three_ways(solve, **kw):
    """One launch per check period, the default's shorter launches, and two
    plain launches per iteration."""
    return solve(cluster_chunks=1, **kw), solve(**kw), solve(use_graphs=0, **kw)


def rel_err(a, b):
    return float(np.max(np.abs(a - b)) / max(1.0, float(np.max(np.abs(b)))))


@pytest.fixture(scope="module")
def refinery():
    return lpgen.refinery_stack()


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("budget", [1, 40, 57, 400])
def test_fixed_budget_bit_identical(engine, precision, budget):
    lp, _ = lpgen.random_lp()
    kw = dict(max_iterations=budget, polish_on_exit=0, polish_feasibility=0, precision=precision)
    on, cut, plain = three_ways(lambda **k: engine.solve_pdhg(lp, **k), **kw)
    assert on.status == ITERATION_LIMIT and on.iterations == budget
    assert same(on, plain) and same(cut, plain)
    if budget >= 40:
        # Two launches per period of 40 instead of one, or of 80.
        assert on.kernel_launches < cut.kernel_launches
        assert plain.kernel_launches - cut.kernel_launches >= 78 * (budget // 40)
    if precision == 0:
        o = oracle.oracle_solve(lp, **kw)
        assert on.restarts == o.restarts
        assert rel_err(on.x, o.x) < 1e-10 and rel_err(on.y, o.y) < 1e-10


@pytest.mark.parametrize("precision", PRECISIONS)
def test_whole_solves_bit_identical(engine, refinery, precision):
    for lp in (lpgen.random_lp()[0], refinery.case(46), refinery.case(16)):
        on, cut, plain = three_ways(lambda **k: engine.solve_pdhg(lp, **k), tolerance=1e-6,
                                    precision=precision)
        assert on.status == OPTIMAL, on.message
        assert same(on, plain) and same(cut, plain)
        # The 24-period cases take clusters in FP32 alone.
        if precision or lp.num_cols < 2000:
            assert cut.kernel_launches < plain.kernel_launches / 2
        assert oracle.oracle_residual(lp, on.x, on.y).converged(1e-6)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_warp_rows_bit_identical(engine, precision):
    lp = lpgen.long_row_stack().case(3)
    assert 32 < lp.k.row_lengths().max() <= 1024
    kw = dict(max_iterations=600, polish_on_exit=0, polish_feasibility=0, precision=precision)
    on, cut, plain = three_ways(lambda **k: engine.solve_pdhg(lp, **k), **kw)
    assert same(on, plain) and same(cut, plain)
    assert on.kernel_launches < cut.kernel_launches < plain.kernel_launches - 1000


def test_rows_longer_than_1024_not_taken(engine):
    lp = lpgen.long_row_stack(m=2000, n=3000, long_len=2500).case(0)
    kw = dict(max_iterations=200, polish_on_exit=0, polish_feasibility=0)
    on, cut, plain = three_ways(lambda **k: engine.solve_pdhg(lp, **k), **kw)
    assert same(on, plain) and same(cut, plain)
    assert on.kernel_launches == cut.kernel_launches == plain.kernel_launches


def test_stack_tail_bit_identical(engine, refinery):
    sub = lpgen.CaseStack(refinery.base, refinery.names[10:20], refinery.c[10:20],
                          refinery.q[10:20], refinery.lower[10:20], refinery.upper[10:20])
    kw = dict(tolerance=1e-6, precision=PRECISION_FP32, split_stacks=0)
    on, cut, plain = three_ways(lambda **k: engine.solve_case_stack(sub, **k), **kw)
    for k, (a, b, c) in enumerate(zip(on, cut, plain)):
        assert a.status == OPTIMAL, (k, a.message)
        assert same(a, c) and same(b, c), k
    assert cut[0].kernel_launches < plain[0].kernel_launches / 2


def test_invalid_option_rejected(engine):
    lp, _ = lpgen.random_lp()
    with pytest.raises(Exception, match="cluster_chunks"):
        engine.solve_pdhg(lp, cluster_chunks=2, max_iterations=10)
