"""Cluster-resident chunks against plain launches, bit for bit.

options.use_graphs=0 runs every iteration as two plain launches; the default
takes the cluster kernel where the matrix is small enough. Both sum every row
in the same order and take the same steps, so x, y and the restart counts are
equal exactly, in both precisions, on:
- matrices with fewer rows than a cluster has CTAs, with one row, with empty
  rows and columns, and at and beyond what the CTAs' threads hold;
- stacks of 2 cases up to more than the device keeps resident;
- rows summed by warps (single LP) and in several segments (stack);
- single LPs and stacks on both sides of every limit, with the route asserted
  by the launches counted, stacks on clusters of 8 CTAs among them;
- budgets that end inside a launch, and the averaged and KKT-restart schemes.
"""
import numpy as np
import pytest

from anukulan_b200 import lpgen
from anukulan_b200.abi import PRECISION_FP32
from anukulan_b200.model import Csr, StandardLp

pytestmark = pytest.mark.gpu

PRECISIONS = [0, PRECISION_FP32]


def small_lp(m, n, seed=3, num_eq=0):
    """A dense-ish boxed LP; the last row and the first column are empty when
    there is room for it."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((m, n)) * (rng.random((m, n)) < 0.5)
    a[0, -1] = 1.0
    if m > 2 and n > 2:
        a[-1, :] = 0.0
        a[:, 0] = 0.0
    r, c = np.nonzero(a)
    k = Csr.from_triplets(m, n, r, c, a[r, c])
    q = a @ rng.uniform(0.0, 1.0, n)
    q[num_eq:] -= 0.1
    return StandardLp(k, rng.standard_normal(n), q, np.zeros(n), np.full(n, 3.0), num_eq, 1.0, 0.0,
                      np.arange(m, dtype=np.int32), np.ones(m), f"small_{m}x{n}")


def same(a, b):
    return (a.iterations == b.iterations and a.restarts == b.restarts
            and np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y))


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape", [(1, 1), (1, 3), (3, 5), (17, 9), (40, 130), (330, 500)])
def test_small_shapes(engine, precision, shape):
    lp = small_lp(*shape, num_eq=shape[0] // 3)
    kw = dict(max_iterations=77, polish_on_exit=0, polish_feasibility=0, precision=precision)
    cluster = engine.solve_pdhg(lp, **kw)
    plain = engine.solve_pdhg(lp, use_graphs=0, **kw)
    assert same(cluster, plain)
    if precision or lp.k.nnz <= 28_000:
        assert plain.kernel_launches - cluster.kernel_launches >= 140


# rows, columns, nonzeros per column, check period, whether FP64 and FP32 take
# clusters.
ROUTES = [(1000, 1500, 8, 40, True, True), (2000, 4096, 4, 40, True, True),
          (2000, 4100, 4, 40, False, True), (1700, 3500, 8, 40, True, True),
          (1700, 3504, 8, 40, False, True), (4000, 8190, 4, 40, False, True),
          (4000, 8200, 4, 40, False, False), (1000, 1500, 8, 5, True, True),
          (1000, 1500, 8, 4, False, False)]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("route", ROUTES)
def test_single_lp_routes(engine, precision, route):
    m, n, per_col, period, fp64, fp32 = route
    lp, _ = lpgen.sparse_random_lp(m, n, per_col)
    kw = dict(max_iterations=120, polish_on_exit=0, polish_feasibility=0, precision=precision,
              termination_check_frequency=period)
    r, plain = engine.solve_pdhg(lp, **kw), engine.solve_pdhg(lp, use_graphs=0, **kw)
    assert same(r, plain)
    # A cluster launch takes the place of at least kClusterLenMin iterations.
    saved = plain.kernel_launches - r.kernel_launches
    assert saved >= 120 if (fp32 if precision else fp64) else saved < 20


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("cols", [8190, 8192, 8200])
def test_largest_shapes(engine, precision, cols):
    # 16 CTAs of 512 threads hold 8,192 columns at best.
    lp, _ = lpgen.sparse_random_lp(cols // 2, cols, 3)
    kw = dict(max_iterations=81, polish_on_exit=0, polish_feasibility=0, precision=precision)
    assert same(engine.solve_pdhg(lp, **kw), engine.solve_pdhg(lp, use_graphs=0, **kw))


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("cases", [2, 7, 14, 15, 29])
def test_stacks(engine, precision, cases):
    stack = lpgen.refinery_stack(periods=5)
    pick = slice(0, cases)
    sub = lpgen.CaseStack(stack.base, stack.names[pick], stack.c[pick], stack.q[pick],
                          stack.lower[pick], stack.upper[pick])
    kw = dict(max_iterations=95, polish_on_exit=0, polish_feasibility=0, precision=precision)
    res = engine.solve_case_stack(sub, **kw)
    plain = engine.solve_case_stack(sub, use_graphs=0, **kw)
    assert all(same(a, b) for a, b in zip(res, plain))
    assert plain[0].kernel_launches - res[0].kernel_launches >= 150


# Refinery periods, cases, precision, whether they take clusters. The device
# keeps 7 clusters of 16 CTAs resident for FP64 plans of this size: 12 cases are
# past four for every three of them, so they take clusters of 8; so do 8 cases,
# which those serve at once. 24 periods leave no room for clusters of 8.
STACK_ROUTES = [(16, 7, 0, True), (16, 8, 0, True), (16, 12, 0, True), (24, 8, 0, True),
                (24, 10, 0, False), (18, 15, PRECISION_FP32, True),
                (24, 15, PRECISION_FP32, True), (24, 24, PRECISION_FP32, False)]


@pytest.mark.parametrize("route", STACK_ROUTES)
def test_stack_routes(engine, route):
    periods, cases, precision, clusters = route
    stack = lpgen.refinery_stack(periods=periods)
    sub = lpgen.CaseStack(stack.base, stack.names[:cases], stack.c[:cases], stack.q[:cases],
                          stack.lower[:cases], stack.upper[:cases])
    kw = dict(max_iterations=121, polish_on_exit=0, polish_feasibility=0, precision=precision,
              split_stacks=0)
    res = engine.solve_case_stack(sub, **kw)
    plain = engine.solve_case_stack(sub, use_graphs=0, **kw)
    assert all(same(a, b) for a, b in zip(res, plain))
    saved = plain[0].kernel_launches - res[0].kernel_launches
    assert saved >= 200 if clusters else saved < 20


@pytest.mark.parametrize("precision", PRECISIONS)
def test_rows_of_several_segments(engine, precision):
    stack = lpgen.long_row_stack(cases=5)  # three rows of 700 nonzeros
    kw = dict(max_iterations=120, polish_on_exit=0, polish_feasibility=0, precision=precision)
    res = engine.solve_case_stack(stack, **kw)
    plain = engine.solve_case_stack(stack, use_graphs=0, **kw)
    assert all(same(a, b) for a, b in zip(res, plain))
    assert plain[0].kernel_launches - res[0].kernel_launches >= 200


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("scheme", [dict(halpern=0), dict(halpern=0, restart_on_fixed_point=0),
                                    dict(pid_primal_weight=0), dict(reflection=0.0),
                                    dict(restarts=0), dict(termination_check_frequency=1),
                                    dict(termination_check_frequency=97)])
def test_schemes(engine, precision, scheme):
    lp, _ = lpgen.random_lp(200, 300)
    kw = dict(max_iterations=200, polish_on_exit=0, polish_feasibility=0, precision=precision)
    kw.update(scheme)
    assert same(engine.solve_pdhg(lp, **kw), engine.solve_pdhg(lp, use_graphs=0, **kw))
