"""Parity of the sm_100a engine against the oracle (the restated reference
PDHG path) and the reference's golden fixtures, through the C ABI.

Tolerances (FP64 engine): the engine runs the reference's arithmetic without
FMA contraction, but sums reductions as trees where the reference sums
serially, so iterates agree to ~1e-12 relative and iteration counts agree
exactly on these problems (allowed to differ by one check period where a
restart test sits within rounding of its threshold). FP32 engine: every
returned point is re-evaluated in FP64 by the oracle and must meet the
requested relative KKT tolerance.
"""
import os

import numpy as np
import pytest

import lp_cases
import oracle
from anukulan_b200 import lpgen
from anukulan_b200.abi import (ITERATION_LIMIT, OPTIMAL, PRECISION_FP32,
                               PRIMAL_INFEASIBLE)

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "pdhg_golden.npz")
SIMPLEX = os.path.join(os.path.dirname(__file__), "golden", "simplex_objectives.npz")
FP64_ITERATE_RTOL = 1e-10


def rel_err(a, b):
    a = np.asarray(a)
    b = np.asarray(b)
    return float(np.max(np.abs(a - b)) / max(1.0, float(np.max(np.abs(b)))))


@pytest.mark.parametrize("name", sorted(lp_cases.KNOWN))
def test_known_optima_fp64(engine, name):
    builder, objective, x = lp_cases.KNOWN[name]
    lp = lp_cases.standard(builder())
    r = engine.solve_pdhg(lp, tolerance=1e-8)
    o = oracle.oracle_solve(lp, tolerance=1e-8)
    assert r.status == OPTIMAL
    assert abs(r.objective - objective) <= 1e-6 * max(1.0, abs(objective))
    if x is not None:
        np.testing.assert_allclose(r.x, x, atol=1e-5)
    assert r.iterations == o.iterations
    assert r.restarts == o.restarts
    assert rel_err(r.x, o.x) < 1e-9 and rel_err(r.y, o.y) < 1e-9


@pytest.mark.parametrize("name", sorted(lp_cases.KNOWN))
def test_known_optima_fp32(engine, name):
    builder, objective, _ = lp_cases.KNOWN[name]
    lp = lp_cases.standard(builder())
    r = engine.solve_pdhg(lp, tolerance=1e-6, precision=PRECISION_FP32)
    assert r.status == OPTIMAL
    res = oracle.oracle_residual(lp, r.x, r.y)
    assert res.converged(1e-6), res
    assert abs(r.objective - objective) <= 1e-4 * max(1.0, abs(objective))


def test_iterates_after_n_iterations_fp64(engine):
    lp, _ = lpgen.random_lp()
    for n_it in (40, 200, 1000):
        kw = dict(max_iterations=n_it, polish_on_exit=0, polish_feasibility=0)
        r = engine.solve_pdhg(lp, **kw)
        o = oracle.oracle_solve(lp, **kw)
        assert r.status == o.status == ITERATION_LIMIT
        assert r.iterations == o.iterations == n_it
        assert r.restarts == o.restarts
        assert rel_err(r.x, o.x) < FP64_ITERATE_RTOL, n_it
        assert rel_err(r.y, o.y) < FP64_ITERATE_RTOL, n_it


def test_random_lp_full_solve_fp64_matches_golden(engine):
    g = np.load(GOLDEN)
    lp, obj = lpgen.random_lp()
    r = engine.solve_pdhg(lp, tolerance=1e-6)
    assert r.status == OPTIMAL
    assert abs(r.iterations - int(g["random_1000x1500/iterations"])) <= 40
    assert abs(r.objective - float(g["random_1000x1500/objective"])) <= 1e-9 * abs(obj)
    assert abs(r.objective - obj) <= 1e-5 * abs(obj)
    simplex = float(np.load(SIMPLEX)["random_1000x1500/objective"])
    assert abs(r.objective - simplex) <= 1e-6 * max(1.0, abs(simplex))


def test_random_lp_fp32_reaches_tolerance(engine):
    lp, obj = lpgen.random_lp()
    r = engine.solve_pdhg(lp, tolerance=1e-6, precision=PRECISION_FP32)
    assert r.status == OPTIMAL, r.message
    res = oracle.oracle_residual(lp, r.x, r.y)
    assert res.converged(1e-6), res
    assert abs(r.objective - obj) <= 1e-5 * abs(obj)
    simplex = float(np.load(SIMPLEX)["random_1000x1500/objective"])
    assert abs(r.objective - simplex) <= 1e-6 * max(1.0, abs(simplex))


@pytest.mark.parametrize("tol", [1e-6, 1e-8])
def test_fp32_refinement_tracks_fp64(engine, tol):
    """FP32 offsets on an FP64 base, re-formed at every check, follow the FP64
    trajectory: same status, iteration count within one check period per
    thousand iterations, objective within the tolerance, and the oracle's
    FP64 residual of the returned point meets the tolerance."""
    lp, obj = lpgen.random_lp()
    a = engine.solve_pdhg(lp, tolerance=tol)
    b = engine.solve_pdhg(lp, tolerance=tol, precision=PRECISION_FP32)
    assert a.status == b.status == OPTIMAL
    assert abs(a.iterations - b.iterations) <= 40 * (1 + a.iterations // 1000)
    assert b.refinement_rounds > 0
    assert oracle.oracle_residual(lp, b.x, b.y).converged(tol)
    assert abs(a.objective - b.objective) <= 10 * tol * abs(a.objective)


@pytest.mark.parametrize("tol", [1e-10, 1e-12, 1e-14])
@pytest.mark.parametrize("which", ["refinery", "random"])
def test_fp32_refinement_reaches_machine_precision(engine, tol, which):
    """Re-centring refinement carries FP32 iterates to FP64 accuracy: on the
    refinery base LP and the 1000x1500 LP the FP32 solve reaches relative KKT
    1e-10, 1e-12 and 1e-14, which plain FP32 iterates cannot (they floor near
    1e-5), and the oracle's FP64 residual of the returned point meets the
    tolerance. The iteration count stays close to the FP64 solve's (measured:
    equal to 1e-12 on both, within 4% at 1e-14 on the refinery; the FP32 run
    is faster at 1e-14 on the random LP)."""
    lp = lpgen.refinery_stack().base if which == "refinery" else lpgen.random_lp()[0]
    a = engine.solve_pdhg(lp, tolerance=tol, max_iterations=400_000)
    b = engine.solve_pdhg(lp, tolerance=tol, precision=PRECISION_FP32, max_iterations=400_000)
    assert a.status == b.status == OPTIMAL, (a.message, b.message)
    assert oracle.oracle_residual(lp, b.x, b.y).converged(tol)
    assert b.iterations <= 1.1 * a.iterations + 40


def test_fp32_plain_without_refinement_runs(engine):
    lp, _ = lpgen.random_lp(300, 450, 8, seed=4)
    r = engine.solve_pdhg(lp, tolerance=1e-4, precision=PRECISION_FP32, refinement=0)
    assert r.status == OPTIMAL and r.refinement_rounds == 0


def test_iteration_limit_exact(engine):
    lp = lp_cases.standard(lp_cases.wyndor())
    r = engine.solve_pdhg(lp, tolerance=1e-14, max_iterations=80,
                          termination_check_frequency=40)
    assert r.status == ITERATION_LIMIT and r.iterations == 80


def test_infeasible_detected(engine):
    r = engine.solve_pdhg(lp_cases.standard(lp_cases.infeasible()), tolerance=1e-8)
    assert r.status == PRIMAL_INFEASIBLE


def test_empty_matrix(engine):
    r = engine.solve_pdhg(lp_cases.standard(lp_cases.empty_rows()), tolerance=1e-8)
    np.testing.assert_allclose(r.x, [0.0, 5.0], atol=1e-6)
    assert abs(r.objective + 5.0) <= 1e-6


def test_deterministic(engine):
    lp, _ = lpgen.random_lp(300, 450, 8, seed=4)
    a = engine.solve_pdhg(lp)
    b = engine.solve_pdhg(lp)
    assert a.iterations == b.iterations and a.restarts == b.restarts
    assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)


def test_warm_start_is_used(engine):
    lp = lp_cases.standard(lp_cases.wyndor())
    cold = engine.solve_pdhg(lp, tolerance=1e-8)
    warm = engine.solve_pdhg(lp, tolerance=1e-8, warm_x=cold.x, warm_y=cold.y,
                             ruiz_iterations=0, pock_chambolle=0)
    assert warm.status == OPTIMAL and warm.iterations < cold.iterations


OPTION_SETS = [
    dict(halpern=0),
    dict(restart_on_fixed_point=0),
    dict(pid_primal_weight=0),
    dict(restarts=0, max_iterations=20000),
    dict(tolerance=1e-8, gap_tolerance=1e-2),
    dict(reuse_products=0),
    dict(constant_step_size=0, max_iterations=2000),
    dict(halpern_restart=1, max_iterations=2000),
    dict(ruiz_iterations=0, pock_chambolle=0),
    dict(use_graphs=0),
]


@pytest.mark.parametrize("opts", OPTION_SETS,
                         ids=lambda d: ",".join(f"{k}={v}" for k, v in d.items()))
def test_option_configurations_match_oracle(engine, opts):
    lp, _ = lpgen.random_lp(300, 450, 8, seed=11)
    r = engine.solve_pdhg(lp, **opts)
    o = oracle.oracle_solve(lp, **opts)
    assert r.status == o.status
    assert abs(r.iterations - o.iterations) <= 40
    if o.status == OPTIMAL:
        assert abs(r.objective - o.objective) <= 1e-6 * max(1.0, abs(o.objective))


def test_evaluate_residual_matches_oracle(engine):
    lp, _ = lpgen.random_lp(300, 450, 8, seed=5)
    rng = np.random.default_rng(3)
    x = rng.uniform(0, 10, lp.num_cols)
    y = rng.standard_normal(lp.num_rows)
    a = engine.evaluate_residual(lp, x, y)
    b = oracle.oracle_residual(lp, x, y)
    for f in ("relative_primal", "relative_dual", "relative_gap", "primal_objective",
              "dual_objective", "primal_residual_inf", "dual_residual_inf"):
        assert abs(getattr(a, f) - getattr(b, f)) <= 1e-12 * max(1.0, abs(getattr(b, f))), f


def test_matrix_norm_matches_oracle(engine):
    lp = lp_cases.standard(lp_cases.norm_4())
    assert abs(engine.estimate_matrix_norm(lp, 500, 1e-12) - 4.0) <= 1e-6
    lp2, _ = lpgen.random_lp(300, 450, 8, seed=5)
    a = engine.estimate_matrix_norm(lp2)
    b = oracle.oracle_matrix_norm(lp2)
    assert abs(a - b) <= 1e-12 * b


def test_invalid_lp_rejected(engine):
    lp = lp_cases.standard(lp_cases.wyndor())
    bad = lp.with_vectors(lower=np.array([1.0, 0.0]), upper=np.array([0.0, 1.0]))
    with pytest.raises(engine.EngineError) as e:
        engine.solve_pdhg(bad)
    assert e.value.code == 1


# ---------------------------------------------------------------- case stack


@pytest.fixture(scope="module")
def stack():
    return lpgen.refinery_stack()


def test_case_stack_fp64_matches_golden(engine, stack):
    g = np.load(GOLDEN)
    res = engine.solve_case_stack(stack, tolerance=1e-6)
    assert len(res) == 60
    for k in (0, 33, 45, 55):
        name = f"refinery_case{k}"
        assert res[k].status == OPTIMAL
        assert abs(res[k].iterations - int(g[f"{name}/iterations"])) <= 80, k
        ref_obj = float(g[f"{name}/objective"])
        assert abs(res[k].objective - ref_obj) <= 1e-7 * abs(ref_obj), k
    for k, r in enumerate(res):
        assert r.status == OPTIMAL, (k, r.message)


def test_case_stack_fp32_reaches_tolerance(engine, stack):
    res = engine.solve_case_stack(stack, tolerance=1e-6, precision=PRECISION_FP32)
    g = np.load(GOLDEN)
    for k, r in enumerate(res):
        assert r.status == OPTIMAL, (k, r.message)
        if k in (0, 33, 45, 55):
            res_k = oracle.oracle_residual(stack.case(k), r.x, r.y)
            assert res_k.converged(1e-6), (k, res_k)
            ref_obj = float(g[f"refinery_case{k}/objective"])
            assert abs(r.objective - ref_obj) <= 1e-5 * abs(ref_obj)


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_case_stack_objectives_match_simplex(engine, stack, precision):
    # The objective oracle: the reference's dual simplex on every one of the
    # 60 cases (tests/golden/simplex_objectives.npz). Relative KKT 1e-6 bounds
    # the duality gap by 1e-6 (1 + |c'x| + |q'y|), about 2e-6 of the
    # objective, so each case is held to 2e-6 relative. The reference's own
    # PDHG at 1e-6 puts 59 of the 60 within 1e-6 (case 46, a demand cut, at
    # 1.30e-6). In FP64 the engine lands on the reference's objectives (1e-9),
    # so on the same single case beyond 1e-6. FP32 iterates round
    # differently, and which cases end between 1e-6 and 2e-6 moves with the
    # kernels' summation order; there only the 2e-6 bound is held.
    g = np.load(SIMPLEX)
    res = engine.solve_case_stack(stack, tolerance=1e-6, precision=precision)
    beyond = []
    for k, r in enumerate(res):
        assert r.status == OPTIMAL, (k, r.message)
        ref_obj = float(g["refinery/objective"][k])
        rel = abs(r.objective - ref_obj) / max(1.0, abs(ref_obj))
        assert rel <= 2e-6, (k, r.objective, ref_obj)
        if rel > 1e-6:
            beyond.append(k)
        if precision == 0:
            # FP64: the reference PDHG's own objective at 1e-6, case by case.
            pd = float(g["refinery/pdhg_objective"][k])
            assert abs(r.objective - pd) <= 1e-9 * abs(pd), (k, r.objective, pd)
    if precision == 0:
        assert beyond == [46], beyond


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_case_stack_objectives_within_1e6_of_simplex(engine, stack, precision):
    # The bench's stack settings: relative KKT 1e-6 with the duality gap held
    # to 5e-7. The gap is relative to 1 + |c'x| + |q'y|, about twice the
    # objective, so this holds every one of the 60 objectives within 1e-6 of
    # the dual simplex optimum, case 46 included (the reference's PDHG at
    # these settings: at most 7.3e-7), at the same iteration count for the
    # hardest case.
    g = np.load(SIMPLEX)
    res = engine.solve_case_stack(stack, tolerance=1e-6, gap_tolerance=5e-7,
                                  precision=precision)
    for k, r in enumerate(res):
        assert r.status == OPTIMAL, (k, r.message)
        assert r.residual.relative_gap <= 5e-7
        ref_obj = float(g["refinery/objective"][k])
        assert abs(r.objective - ref_obj) <= 1e-6 * abs(ref_obj), (k, r.objective, ref_obj)


def test_case_stack_tail_compaction(engine, stack):
    # An FP32 stack compacts its per-case arrays to its last running case,
    # which then takes the single-LP kernels: 64 cases (the 60, then cases
    # 0-3 again), one stack. Every case must come back in its own
    # slot with its own answer: the objective of its simplex golden to 1e-6,
    # the duplicates equal to their originals, every returned point converged
    # in FP64 (sampled), and the hardest case - the one that finishes in the
    # compacted layout - within two check periods of its separate solve.
    g = np.load(SIMPLEX)["refinery/objective"]
    idx = list(range(60)) + [0, 1, 2, 3]
    sub = _rolling(stack, idx)
    res = engine.solve_case_stack(sub, tolerance=1e-6, gap_tolerance=5e-7,
                                  precision=PRECISION_FP32, split_stacks=0)
    assert len(res) == 64
    for slot, (k, r) in enumerate(zip(idx, res)):
        assert r.status == OPTIMAL, (slot, r.message)
        assert abs(r.objective - g[k]) <= 1e-6 * abs(g[k]), (slot, r.objective, g[k])
    for dup in range(4):
        assert res[60 + dup].iterations == res[dup].iterations
        assert abs(res[60 + dup].objective - res[dup].objective) <= 1e-9 * abs(res[dup].objective)
    hard = int(np.argmax([r.iterations for r in res]))
    for slot in (hard, 5, 33, 47):
        rr = oracle.oracle_residual(stack.case(idx[slot]), res[slot].x, res[slot].y)
        assert rr.converged(1e-6), (slot, rr)
    alone = engine.solve_pdhg(stack.case(idx[hard]), tolerance=1e-6, gap_tolerance=5e-7,
                              precision=PRECISION_FP32)
    assert abs(alone.iterations - res[hard].iterations) <= 80, (alone.iterations, res[hard].iterations)


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_case_stack_graphs_bit_identical(engine, stack, precision):
    # Iteration chunks, termination checks and re-centrings replayed as CUDA
    # graphs run the same kernels on the same buffers as direct launches:
    # 44 cases (two half-stacks, too many for clusters), results identical bit
    # for bit.
    sub = _rolling(stack, list(range(44)))
    kw = dict(tolerance=1e-6, precision=precision)
    graphs = engine.solve_case_stack(sub, use_graphs=1, **kw)
    direct = engine.solve_case_stack(sub, use_graphs=0, **kw)
    for k, (a, b) in enumerate(zip(graphs, direct)):
        assert a.status == b.status == OPTIMAL, (k, a.message)
        assert a.iterations == b.iterations and a.restarts == b.restarts, k
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y), k
    assert graphs[0].refinement_rounds == direct[0].refinement_rounds


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_single_lp_graphs_bit_identical(engine, precision):
    # Too many columns for a cluster: iterations are graph-captured launches.
    lp, _ = lpgen.sparse_random_lp(6000, 9000, 8)
    kw = dict(max_iterations=250, polish_on_exit=0, polish_feasibility=0, precision=precision)
    graphs, direct = engine.solve_pdhg(lp, **kw), engine.solve_pdhg(lp, use_graphs=0, **kw)
    assert graphs.kernel_launches == direct.kernel_launches >= 500
    assert graphs.iterations == direct.iterations and graphs.restarts == direct.restarts
    assert np.array_equal(graphs.x, direct.x) and np.array_equal(graphs.y, direct.y)


def _rolling(stack, idx):
    return lpgen.CaseStack(stack.base, [stack.names[i] for i in idx], stack.c[idx], stack.q[idx],
                           stack.lower[idx], stack.upper[idx])


def test_rolling_stack_fp64_matches_lockstep(engine, stack):
    # 90 cases (the 60 and the first 30 again) exceed one run's 64 slots: the
    # stack rolls, each freed slot admitting the next case at a check. Every
    # case runs its own iteration from its admission, so it must end as in
    # the 60-case lockstep stack.
    idx = list(range(60)) + list(range(30))
    res = engine.solve_case_stack(_rolling(stack, idx), tolerance=1e-6)
    ref = engine.solve_case_stack(stack, tolerance=1e-6)
    assert len(res) == 90
    for i, k in enumerate(idx):
        assert res[i].status == ref[k].status == OPTIMAL, (i, k)
        assert abs(res[i].iterations - ref[k].iterations) <= 80, (i, k)
        assert abs(res[i].objective - ref[k].objective) <= 1e-8 * abs(ref[k].objective), (i, k)


def test_rolling_stack_fp32_admitted_cases_converge(engine, stack):
    idx = list(range(60)) + [16, 33, 45, 55, 0, 7, 21]
    res = engine.solve_case_stack(_rolling(stack, idx), tolerance=1e-6, precision=PRECISION_FP32)
    for i in range(60, len(idx)):
        k = idx[i]
        assert res[i].status == OPTIMAL, (i, res[i].message)
        r = oracle.oracle_residual(stack.case(k), res[i].x, res[i].y)
        assert r.converged(1e-6), (k, r)


@pytest.mark.parametrize("count", [6, 20])
def test_case_stack_warm_start_matches_single(engine, stack, count):
    # Warm starts go to every case as solve_pdhg takes them; 20 cases also
    # exercise the two half-stacks.
    sub = _rolling(stack, list(range(count)))
    cold = engine.solve_case_stack(sub, tolerance=1e-6)
    wx = np.stack([r.x for r in cold])
    wy = np.stack([r.y for r in cold])
    solver = engine.CaseStackSolver(sub.base, sub.c, sub.q, sub.lower, sub.upper, tolerance=1e-6)
    try:
        warm = solver.solve(wx, wy)
    finally:
        solver.close()
    for k in (0, count // 2, count - 1):
        single = engine.solve_pdhg(sub.case(k), warm_x=wx[k], warm_y=wy[k], tolerance=1e-6)
        assert warm[k].status == single.status == OPTIMAL, k
        assert abs(warm[k].iterations - single.iterations) <= 40, k
        assert abs(warm[k].objective - single.objective) <= 1e-8 * abs(single.objective), k


def test_cached_blocks_reused_across_solvers(engine, stack):
    # Each closed solver leaves its blocks in the process-wide cache and the
    # next one takes them: the results of successive create-solve-close
    # cycles (two half-stacks, FP32) must be identical, before and after the
    # cache is released.
    sub = _rolling(stack, list(range(20)))

    def cycle():
        solver = engine.CaseStackSolver(sub.base, sub.c, sub.q, sub.lower, sub.upper,
                                        tolerance=1e-6, precision=PRECISION_FP32)
        try:
            return solver.solve()
        finally:
            solver.close()

    first = cycle()
    again = cycle()
    assert engine.release_cached_memory() > 0
    after = cycle()
    for res in (again, after):
        for a, b in zip(first, res):
            assert a.status == b.status == OPTIMAL
            assert a.iterations == b.iterations
            assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_persistent_chunks_match_graphs(engine, stack, precision):
    # One cooperative launch per chunk runs the same arithmetic in the same
    # order as the two launches per iteration of the graphs: identical
    # iterates, iteration counts and restarts, case by case. In FP32 the
    # graph path hands the stack's last running case to the single-LP
    # kernels once it runs alone (tail compaction; the persistent path does
    # not), so that one case's FP32 sums round differently from there on:
    # same status, iterations and restarts, iterates equal to rounding.
    kw = dict(tolerance=1e-6, precision=precision, split_stacks=0)
    persistent = engine.solve_case_stack(stack, persistent_chunks=1, **kw)
    graphs = engine.solve_case_stack(stack, persistent_chunks=0, **kw)
    last = int(np.argmax([r.iterations for r in graphs]))
    for k, (a, b) in enumerate(zip(persistent, graphs)):
        assert a.status == b.status == OPTIMAL, (k, a.message)
        assert a.iterations == b.iterations and a.restarts == b.restarts, k
        if precision == PRECISION_FP32 and k == last:
            np.testing.assert_allclose(a.x, b.x, rtol=1e-6, atol=1e-6 * np.abs(b.x).max())
            np.testing.assert_allclose(a.y, b.y, rtol=1e-6, atol=1e-6 * np.abs(b.y).max())
        else:
            assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y), k
    assert persistent[0].kernel_launches < graphs[0].kernel_launches


@pytest.mark.parametrize("precision", [0, PRECISION_FP32])
def test_persistent_chunks_long_rows(engine, precision):
    # Rows of 700 nonzeros cut into segments longer than a warp: the chunk
    # kernel reloads the tail of those segments in every phase. A fixed
    # iteration budget, compared bit for bit with the graphs.
    st = lpgen.long_row_stack()
    kw = dict(max_iterations=400, precision=precision, split_stacks=0,
              polish_on_exit=0, polish_feasibility=0)
    persistent = engine.solve_case_stack(st, persistent_chunks=1, **kw)
    graphs = engine.solve_case_stack(st, persistent_chunks=0, **kw)
    for k, (a, b) in enumerate(zip(persistent, graphs)):
        assert a.iterations == b.iterations == 400, k
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y), k
    assert persistent[0].kernel_launches < graphs[0].kernel_launches


def test_case_stack_equals_single_solves(engine, stack):
    sub = lpgen.CaseStack(stack.base, stack.names[:5], stack.c[:5], stack.q[:5],
                          stack.lower[:5], stack.upper[:5])
    batch = engine.solve_case_stack(sub, tolerance=1e-6)
    for k in range(5):
        single = engine.solve_pdhg(stack.case(k), tolerance=1e-6)
        assert batch[k].status == single.status
        assert abs(batch[k].iterations - single.iterations) <= 40
        assert abs(batch[k].objective - single.objective) <= 1e-8 * abs(single.objective)


# ------------------------------------------------------------- backend seam


def test_backend_seam_contract(engine):
    import ctypes as C
    L = engine.lib()
    rng = np.random.default_rng(20260830)
    n, m = 733, 501

    def dev(v):
        p = C.c_void_p()
        engine.check(L.anu_backend_allocate(len(v), C.byref(p)))
        a = np.ascontiguousarray(v, np.float64)
        engine.check(L.anu_backend_upload(a.ctypes.data_as(C.POINTER(C.c_double)), p, len(v)))
        return p

    def host(p, count):
        out = np.zeros(count)
        engine.check(L.anu_backend_download(p, out.ctypes.data_as(C.POINTER(C.c_double)), count))
        return out

    x = rng.uniform(-1, 1, n)
    c = rng.standard_normal(n)
    kty = rng.standard_normal(n)
    lo = np.full(n, -0.5)
    hi = np.full(n, 0.5)
    anchor = rng.standard_normal(n)
    px, pc, pk, pl, ph, pa = map(dev, (x, c, kty, lo, hi, anchor))
    xo, dxo, xbo = dev(np.zeros(n)), dev(np.zeros(n)), dev(np.zeros(n))
    tau, gamma, w = 0.3, 1.0, 0.75
    engine.check(L.anu_backend_primal_update(n, tau, gamma, w, px, pc, pk, pl, ph, pa, xo, dxo, xbo))
    v = np.clip(x - tau * (c - kty), lo, hi)
    d = v - x
    nxt = w * (v + gamma * d) + (1 - w) * anchor
    assert np.array_equal(host(dxo, n), d)
    assert np.array_equal(host(xbo, n), v + d)
    assert np.array_equal(host(xo, n), nxt)
    # dot / norms
    out = C.c_double()
    engine.check(L.anu_backend_dot(px, pc, n, C.byref(out)))
    assert abs(out.value - float(np.dot(x, c))) <= 1e-13 * np.abs(x * c).sum()
    engine.check(L.anu_backend_inf_norm(pc, n, C.byref(out)))
    assert out.value == float(np.max(np.abs(c)))
    # sparse product, ragged rows, every 5th row empty
    r, cc, vv = [], [], []
    for i in range(m):
        if i % 5 == 0:
            continue
        length = 2 + (i * 7) % 40 if i % 100 else 3000
        cols = rng.choice(n, size=min(length, n), replace=False)
        r += [i] * len(cols)
        cc += list(cols)
        vv += list(rng.standard_normal(len(cols)))
    from anukulan_b200.model import Csr
    from anukulan_b200.abi import anu_csr
    a = Csr.from_triplets(m, n, r, cc, vv)
    st = np.ascontiguousarray(a.start, np.int32)
    ix = np.ascontiguousarray(a.index, np.int32)
    va = np.ascontiguousarray(a.value, np.float64)
    csr = anu_csr(m, n, a.nnz, st.ctypes.data_as(C.POINTER(C.c_int32)),
                  ix.ctypes.data_as(C.POINTER(C.c_int32)),
                  va.ctypes.data_as(C.POINTER(C.c_double)))
    engine.check(L.anu_backend_prepare(12345, C.byref(csr)))
    py = dev(np.zeros(m))
    engine.check(L.anu_backend_multiply(12345, px, py))
    want = np.array([sum(a.value[k] * x[a.index[k]] for k in range(a.start[i], a.start[i + 1]))
                     for i in range(m)])
    got = host(py, m)
    assert np.max(np.abs(got - want)) <= 1e-13 * max(1.0, np.max(np.abs(want)))
    engine.check(L.anu_backend_release())
    for p in (px, pc, pk, pl, ph, pa, xo, dxo, xbo, py):
        engine.check(L.anu_backend_deallocate(p))
