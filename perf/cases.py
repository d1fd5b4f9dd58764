"""The work users have this engine do, as timed cases.

Each case goes through the package's public entry points: the one-call solve,
prepared handles, case stacks, packed batches, the unrolled program with its
adjoint, and the backend seam's coarse operations. Sizes span the workloads
of ``anukulan_b200.lpgen``: 1,000 to 200,000 rows for single LPs, refinery
plans of 2 to 24 periods, 1 to 64 cases in a stack.

Solves that run a fixed budget of iterations (``iterations`` in the case) are
what branch-and-bound nodes, crossover seeds and rolling re-solves ask for,
and their length does not depend on the data.
"""
import itertools
import math

import numpy as np
import torch

from anukulan_b200 import lpgen, pdhg
from anukulan_b200.abi import PRECISION_FP32, PRECISION_FP64
from anukulan_b200.model import Csr, StandardLp, to_standard_form

CHECK_EVERY = 40  # the default termination_check_frequency
PER_COL = 8       # nonzeros per column of the random and power-law LPs
BUDGET = dict(tolerance=1e-9, polish_feasibility=False, polish_on_exit=False,
              time_limit_seconds=300.0)


def listed():
    return [
        # The reference's own solver over this library's backend: one PDHG
        # iteration is four coarse operations on device vectors. The small LP
        # is bound by launches, the large one by memory.
        dict(name="seam_iteration_small", kind="seam", lp="random", rows=1000),
        dict(name="seam_iteration_large", kind="seam", lp="powerlaw", rows=200_000),
        # The same solver's termination check: fresh products and the seven
        # convergence terms, read back by the host.
        dict(name="seam_check_ragged", kind="seam_check", lp="powerlaw", rows=37_501),
        # A whole default solve, set-up included, of the plain FP64 workload.
        dict(name="solve_small_fp64", kind="solve", lp="random", rows=1000, tolerance=1e-4),
        # A prepared planning LP re-solved with new prices and demands.
        dict(name="resolve_refinery_fp32", kind="resolve", lp="refinery", periods=24,
             precision="fp32", iterations=2000),
        # Large single LPs, both precisions.
        dict(name="run_powerlaw_fp32", kind="run", lp="powerlaw", rows=200_000,
             precision="fp32", iterations=1200),
        dict(name="run_powerlaw_fp64", kind="run", lp="powerlaw", rows=60_007,
             precision="fp64", iterations=1200),
        # The what-if stack of the planning LP.
        dict(name="stack_refinery_60_fp32", kind="stack", periods=24, cases=60,
             precision="fp32", iterations=2000),
        # A handful of branch-and-bound nodes: FP64 bounds, few cases.
        dict(name="stack_nodes_7_fp64", kind="stack", periods=10, cases=7,
             precision="fp64", iterations=1200),
        # What-if sensitivities of the whole stack, forward and backward. At
        # this length FP32 gradients are still those of the FP64 program; over
        # thousands of steps a projection's kink can flip one by its own size.
        dict(name="unrolled_60_fp32", kind="unrolled", periods=24, cases=60,
             precision="fp32", iterations=300, checkpoint=100),
        # One plan's sensitivity in FP64, a length the checkpoints do not divide.
        dict(name="unrolled_1_fp64", kind="unrolled", periods=6, cases=1,
             precision="fp64", iterations=450, checkpoint=64),
        # Unequal independent LPs, several in flight.
        dict(name="packed_16_fp32", kind="packed", count=16, min_rows=500, max_rows=20_000,
             precision="fp32", iterations=1000, workers=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["seam", "seam_check", "solve", "resolve", "run", "run", "stack", "stack",
                       "unrolled", "unrolled", "packed"])
    precision = rng.choice(["fp32", "fp64"])
    if kind in ("seam", "seam_check"):
        return dict(kind=kind, lp=rng.choice(["random", "powerlaw"]),
                    rows=_log_int(rng, 1000, 200_000))
    if kind == "solve":
        return dict(kind=kind, lp="random", rows=_log_int(rng, 500, 3000), tolerance=1e-4)
    if kind == "resolve":
        return dict(kind=kind, lp="refinery", periods=rng.randint(2, 24), precision=precision,
                    iterations=rng.randint(200, 2000))
    if kind == "run":
        return dict(kind=kind, lp=rng.choice(["random", "powerlaw"]),
                    rows=_log_int(rng, 1000, 120_000), precision=precision,
                    iterations=rng.randint(200, 1200))
    if kind == "stack":
        return dict(kind=kind, periods=rng.randint(2, 24), cases=rng.randint(2, 64),
                    precision=precision, iterations=rng.randint(200, 1000))
    if kind == "unrolled":
        return dict(kind=kind, periods=rng.randint(2, 24), cases=_log_int(rng, 1, 64),
                    precision=precision,
                    iterations=rng.randint(60, 300 if precision == "fp32" else 600),
                    checkpoint=rng.randint(20, 120))
    return dict(kind="packed", count=rng.randint(3, 14), min_rows=500, max_rows=12_000,
                precision=precision, iterations=rng.randint(200, 800),
                workers=rng.choice([4, 8]))


# ------------------------------------------------------------------ inputs


def _rng(seed, stream):
    return np.random.default_rng([seed & 0x7FFFFFFF, stream])


def _planted(k, rng, name):
    """c and q of a known primal-dual optimum (x0, y0): columns at zero with
    probability 0.3, bounds [0, 10], all rows equalities."""
    x0 = rng.uniform(0.0, 10.0, k.cols)
    zero = rng.random(k.cols) < 0.3
    x0[zero] = 0.0
    y0 = rng.standard_normal(k.rows)
    slack = np.where(zero, np.abs(rng.standard_normal(k.cols)), 0.0)
    rows_of = np.repeat(np.arange(k.rows), np.diff(k.start))
    q = np.bincount(rows_of, weights=k.value * x0[k.index], minlength=k.rows)
    c = np.bincount(k.index, weights=k.value * y0[rows_of], minlength=k.cols) + slack
    lp = StandardLp(k, c, q, np.zeros(k.cols), np.full(k.cols, 10.0), k.rows, 1.0, 0.0,
                    np.arange(k.rows, dtype=np.int32), np.ones(k.rows), name)
    return lp, x0, y0


def _sparse_lp(shape, rows, seed):
    """A planted LP with 8 nonzeros per column, 1.5 columns per row. "random":
    uniform rows; "powerlaw": row lengths from P(L) ~ L^-2.2 on [3, 5000]."""
    rng = _rng(seed, 1)
    cols = (3 * rows) // 2
    if shape == "powerlaw":
        support = np.arange(3, min(5000, max(4, cols // 4)) + 1)
        p = support.astype(np.float64) ** -2.2
        lengths = rng.choice(support, size=rows, p=p / p.sum())
        slots = np.repeat(np.arange(rows), lengths)
        total = cols * PER_COL
        if slots.size < total:
            slots = np.concatenate([slots, rng.integers(0, rows, total - slots.size)])
        else:
            slots = rng.permutation(slots)
        slots = rng.permutation(slots[:total]).reshape(cols, PER_COL)
    else:
        slots = rng.integers(0, rows, size=(cols, PER_COL))
    slots.sort(axis=1)
    while True:  # a row at most once in a column
        twice = np.zeros(slots.shape, bool)
        twice[:, 1:] = slots[:, 1:] == slots[:, :-1]
        count = int(twice.sum())
        if count == 0:
            break
        slots[twice] = rng.integers(0, rows, count)
        slots.sort(axis=1)
    flat = slots.reshape(-1)
    order = np.argsort(flat, kind="stable")
    start = np.concatenate([[0], np.cumsum(np.bincount(flat, minlength=rows))]).astype(np.int32)
    k = Csr(rows, cols, start, (order // PER_COL).astype(np.int32),
            rng.standard_normal(flat.size))
    return _planted(k, rng, f"{shape}_{rows}x{cols}")


def _refinery(periods, seed):
    model, layout = lpgen.refinery_model(periods, seed=seed & 0x7FFFFFFF)
    form = to_standard_form(model)
    return form.lp, layout


def _what_ifs(lp, layout, count, seed):
    """c, q and upper of `count` what-if cases: a crude's price moved by up to
    6%, a supply bound halved, or a demand or capacity moved by up to 20%."""
    rng = _rng(seed, 2)
    c, q, upper = (np.repeat(v[None, :], count, 0) for v in (lp.c, lp.q, lp.upper))
    movable = np.flatnonzero(lp.q != 0.0)
    for k in range(count):
        buy = np.arange(layout.periods) * layout.cols_per_period + int(rng.integers(layout.crudes))
        what = k % 3
        if what == 0:
            c[k, buy] *= 1.0 + rng.uniform(-0.06, 0.06)
        elif what == 1:
            upper[k, buy] *= 0.5
        else:
            q[k, rng.choice(movable, layout.periods, replace=False)] *= rng.uniform(0.8, 1.0)
    return c, q, upper


def _stack_inputs(case, seed):
    lp, layout = _refinery(case["periods"], seed)
    c, q, upper = _what_ifs(lp, layout, case["cases"], seed)
    return lp, c, q, np.repeat(lp.lower[None, :], case["cases"], 0), upper


def _resolve_inputs(case, seed):
    lp, layout = _refinery(case["periods"], seed)
    rng = _rng(seed, 3)
    c = lp.c * (1.0 + 0.03 * rng.standard_normal(lp.c.size))
    q = lp.q * rng.uniform(0.9, 1.0, lp.q.size)
    return lp, c, q


def _packed_sizes(case):
    """Row counts spread evenly over the range's logarithm, odd ones among
    them; the case fixes them, so every seed's batch costs the same."""
    sizes = np.exp(np.linspace(math.log(case["min_rows"]), math.log(case["max_rows"]),
                               case["count"]))
    return [int(s) + (5 * i) % 9 for i, s in enumerate(sizes)]


def _packed_inputs(case, seed):
    return [_sparse_lp("random", m, seed + 7919 * (i + 1))[0]
            for i, m in enumerate(_packed_sizes(case))]


def _precision(case):
    return PRECISION_FP32 if case["precision"] == "fp32" else PRECISION_FP64


def _budget(case):
    return dict(BUDGET, precision=_precision(case), max_iterations=case["iterations"])


_matrix_ids = itertools.count(1 << 40)


def _prepare_matrix(k):
    """`k` on the device under an id of its own, as the backend adapter does."""
    view = pdhg.CLp(StandardLp(k, np.zeros(k.cols), np.zeros(k.rows), np.zeros(k.cols),
                               np.zeros(k.cols), k.rows, 1.0, 0.0,
                               np.arange(k.rows, dtype=np.int32), np.ones(k.rows), ""))
    ident = next(_matrix_ids)
    pdhg.check(pdhg.lib().anu_backend_prepare(ident, view.struct.k))
    return ident


def _seam_vectors(case, seed):
    """One iteration's vectors, part of the way through a solve."""
    lp, x0, y0 = _sparse_lp(case["lp"], case["rows"], seed)
    rng = _rng(seed, 5)
    m, n = lp.k.rows, lp.k.cols
    x = np.clip(x0 + 0.1 * rng.standard_normal(n), 0.0, 10.0)
    y = y0 + 0.1 * rng.standard_normal(m)
    v = dict(x=x, y=y, c=lp.c, q=lp.q, lower=lp.lower, upper=lp.upper,
             anchor=np.clip(x0 + 0.2 * rng.standard_normal(n), 0.0, 10.0),
             anchor_y=y0 + 0.2 * rng.standard_normal(m),
             kx=rng.standard_normal(m), anchor_kx=rng.standard_normal(m),
             row_scale=rng.uniform(0.2, 1.5, m), col_scale=rng.uniform(0.2, 1.5, n))
    return lp, v


TAU, SIGMA, GAMMA, HALPERN = 0.05, 0.04, 1.0, 17.0 / 18.0


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("seam", "seam_check"):
        lp, v = _seam_vectors(case, seed)
        m, n = lp.k.rows, lp.k.cols
        state = {name: torch.from_numpy(a).cuda() for name, a in v.items()}
        state.update(kind=kind, m=m, n=n, num_eq=lp.num_equalities,
                     k=_prepare_matrix(lp.k), kt=_prepare_matrix(lp.k.transpose()))
        for name, size in (("kty", n), ("x_out", n), ("dx", n), ("x_bar", n), ("kx_bar", m),
                           ("y_out", m), ("dy", m), ("k_out", m), ("k_dx", m)):
            state[name] = torch.zeros(size, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return state
    if kind == "solve":
        return dict(kind=kind, lp=_sparse_lp(case["lp"], case["rows"], seed)[0],
                    tolerance=case["tolerance"])
    if kind == "resolve":
        lp, c, q = _resolve_inputs(case, seed)
        return dict(kind=kind, handle=pdhg.PdhgHandle(lp, **_budget(case)), c=c, q=q)
    if kind == "run":
        lp = _sparse_lp(case["lp"], case["rows"], seed)[0]
        # The tile is fixed, as a caller does who has run an LP of this
        # shape: the trials would time a choice, not the work.
        return dict(kind=kind, handle=pdhg.PdhgHandle(
            lp, tile_threads=256 if case["precision"] == "fp32" else 128, **_budget(case)))
    if kind == "stack":
        lp, c, q, lower, upper = _stack_inputs(case, seed)
        return dict(kind=kind,
                    solver=pdhg.CaseStackSolver(lp, c, q, lower, upper, **_budget(case)))
    if kind == "unrolled":
        lp, c, q, lower, upper = _stack_inputs(case, seed)
        price = c * (1.0 + 0.05 * _rng(seed, 6).standard_normal(c.shape))
        return dict(kind=kind, price=price, program=pdhg.UnrolledPdhg(
            lp, c, q, lower, upper, iterations=case["iterations"],
            checkpoint_every=case["checkpoint"], precision=_precision(case)))
    if kind == "packed":
        return dict(kind=kind, solver=pdhg.PackedBatchSolver(
            _packed_inputs(case, seed), workers=case["workers"], tile_threads=128,
            **_budget(case)))
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "seam":
        L, s = pdhg.lib(), state
        p = {name: t.data_ptr() for name, t in s.items() if torch.is_tensor(t)}
        pdhg.check(L.anu_backend_multiply(s["kt"], p["y"], p["kty"]))
        pdhg.check(L.anu_backend_primal_update(
            s["n"], TAU, GAMMA, HALPERN, p["x"], p["c"], p["kty"], p["lower"], p["upper"],
            p["anchor"], p["x_out"], p["dx"], p["x_bar"]))
        pdhg.check(L.anu_backend_multiply(s["k"], p["x_bar"], p["kx_bar"]))
        pdhg.check(L.anu_backend_dual_update(
            s["m"], s["num_eq"], SIGMA, GAMMA, HALPERN, p["y"], p["q"], p["kx_bar"], p["kx"],
            p["anchor_y"], p["anchor_kx"], p["y_out"], p["dy"], p["k_out"], p["k_dx"]))
        return [s[name] for name in ("x_out", "dx", "x_bar", "y_out", "dy", "k_out", "k_dx")]
    if kind == "seam_check":
        L, s = pdhg.lib(), state
        p = {name: t.data_ptr() for name, t in s.items() if torch.is_tensor(t)}
        terms = np.zeros(7)
        pdhg.check(L.anu_backend_multiply(s["k"], p["x"], p["kx_bar"]))
        pdhg.check(L.anu_backend_multiply(s["kt"], p["y"], p["kty"]))
        pdhg.check(L.anu_backend_convergence_terms(
            s["n"], s["m"], p["c"], p["lower"], p["upper"], p["q"], p["row_scale"],
            p["col_scale"], s["num_eq"], p["x"], p["kx_bar"], p["y"], p["kty"],
            pdhg.f64_ptr(terms)))
        return [s["kx_bar"], s["kty"], terms]
    if kind == "solve":
        r = pdhg.solve_pdhg(state["lp"], tolerance=state["tolerance"])
        return [r.x, r.y, r.objective]
    if kind == "resolve":
        state["handle"].set_case(c=state["c"], q=state["q"])
        r = state["handle"].run()
        return [r.x, r.y, r.objective]
    if kind == "run":
        r = state["handle"].run()
        return [r.x, r.y, r.objective]
    if kind == "stack":
        results = state["solver"].solve()
        return [np.stack([r.x for r in results]), np.stack([r.y for r in results]),
                np.array([r.objective for r in results])]
    if kind == "packed":
        return [[r.x, r.y, r.objective] for r in state["solver"].solve()]
    x, y = state["program"].forward()
    grad_c, grad_q = state["program"].backward(state["price"])
    return [x, y, grad_c, grad_q]


# -------------------------------------------------------------------- work


def work(case):
    """Bytes: the matrix once (an FP64 value and a 4-byte index per nonzero,
    the row starts), each case's vectors in and its results out, FP64 as the
    entry points take them. Operations: both products and both steps of every
    iteration, for every case."""
    kind = case["kind"]
    cases = case.get("cases", 1)
    if "periods" in case:
        m, n = 115 * case["periods"], 160 * case["periods"]
        nnz = int(11.55 * n)
    elif kind == "packed":
        m = sum(_packed_sizes(case))
        n = (3 * m) // 2
        nnz = PER_COL * n
    else:
        m = case["rows"]
        n = (3 * m) // 2
        nnz = PER_COL * n
    matrix = 12 * nnz + 4 * (m + 1)
    if kind == "seam":
        # Both orientations are prepared matrices of the call. Vectors: 5 in
        # and 3 out over columns, 5 in and 4 out over rows.
        return dict(bytes=2 * matrix + 4 * (n - m) + 64 * n + 72 * m,
                    flops=4 * nnz + 8 * n + 12 * m)
    if kind == "seam_check":
        return dict(bytes=2 * matrix + 4 * (n - m) + 48 * n + 40 * m,
                    flops=4 * nnz + 14 * n + 10 * m)
    step = cases * (4 * nnz + 12 * n + 14 * m)
    size = matrix + 8 * cases * (4 * n + 2 * m)
    if kind == "solve":
        # Some hundreds of iterations reach 1e-4 at these sizes.
        return dict(bytes=size, flops=400 * step)
    if kind == "unrolled":
        # Forward, the recomputation between checkpoints, and the reverse.
        return dict(bytes=size + 8 * cases * (2 * n + m), flops=3 * case["iterations"] * step)
    return dict(bytes=size, flops=case["iterations"] * step)


# ------------------------------------------------------------------- exact
#
# Plain FP64 torch: the algorithm as published (diagonal scaling, reflected
# Halpern PDHG with restarts and the PID primal weight), on whole vectors.


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_device())


class _Scaled:
    """The scaled matrix of an LP, its scaling and its norm estimate."""

    def __init__(self, k):
        dev = _device()
        row = torch.as_tensor(np.repeat(np.arange(k.rows), np.diff(k.start)), device=dev)
        col = torch.as_tensor(k.index.astype(np.int64), device=dev)
        val = _t(k.value)
        self.m, self.n = k.rows, k.cols
        self.d1, self.d2 = (torch.ones(s, dtype=torch.float64, device=dev)
                            for s in (k.rows, k.cols))
        for sweep in range(11):
            a = val.abs()
            factors = []
            for size, idx in ((k.rows, row), (k.cols, col)):
                norm = torch.zeros(size, dtype=torch.float64, device=dev)
                if sweep < 10:
                    norm.scatter_reduce_(0, idx, a, "amax")
                else:
                    norm.index_add_(0, idx, a)
                factors.append(torch.where(norm > 0, norm, 1.0).rsqrt())
            val = val * factors[0][row] * factors[1][col]
            self.d1 = self.d1 * factors[0]
            self.d2 = self.d2 * factors[1]
        self.k = torch.sparse_coo_tensor(torch.stack([row, col]), val,
                                         (k.rows, k.cols)).coalesce().to_sparse_csr()
        self.kt = torch.sparse_coo_tensor(torch.stack([col, row]), val,
                                          (k.cols, k.rows)).coalesce().to_sparse_csr()
        v = 1.0 + 0.1 * (torch.arange(k.cols, device=dev) % 7).double()
        v = (v / v.norm())[:, None]
        sigma = 0.0
        for it in range(200):
            w = self.kt @ (self.k @ v)
            estimate = math.sqrt(float(w.norm()))
            if it > 0 and abs(estimate - sigma) <= 1e-8 * estimate:
                sigma = estimate
                break
            sigma = estimate
            v = w / w.norm()
        self.norm = sigma


def _exact_solve(lp, c, q, lower, upper, iterations):
    """x, y (cases x length) and objectives after `iterations` of reflected
    Halpern PDHG; c, q, lower, upper are cases x length."""
    s = _Scaled(lp.k)
    c, q, lower, upper = (_t(a).T.contiguous() for a in (c, q, lower, upper))
    d1, d2 = s.d1[:, None], s.d2[:, None]
    cs, qs, lo, hi = c * d2, q * d1, lower / d2, upper / d2
    eta = 0.9 / s.norm
    cn, qn = cs.norm(dim=0), qs.norm(dim=0)
    omega = torch.where((cn > 1e-12) & (qn > 1e-12), cn / qn, 1.0)
    cone = (torch.arange(s.m, device=cs.device) >= lp.num_equalities)[:, None]
    x = torch.zeros_like(cs)
    x = torch.where(x < lo, torch.where(lo.isfinite(), lo, 0.0), x)
    x = torch.where(x > hi, torch.where(hi.isfinite(), hi, 0.0), x)
    y = torch.zeros_like(qs)
    ax, ay = torch.zeros_like(x), torch.zeros_like(y)
    xr, yr = x.clone(), y.clone()
    count = torch.zeros_like(omega)        # steps since the anchor
    since = torch.zeros_like(omega)        # iterations since the restart
    reset = torch.ones_like(omega, dtype=torch.bool)
    at_restart = torch.full_like(omega, math.inf)
    last = torch.full_like(omega, math.inf)
    previous = torch.zeros_like(omega)
    seen = torch.zeros_like(reset)
    for it in range(iterations):
        v = torch.minimum(torch.maximum(x - (eta / omega) * (cs - s.kt @ y), lo), hi)
        dx = v - x
        bar = v + dx
        w = y + (eta * omega) * (qs - s.k @ bar)
        w = torch.where(cone, w.clamp_min(0.0), w)
        dy = w - y
        nx, ny = bar, w + dy
        a = torch.where(reset, 1.0, (count + 1.0) / (count + 2.0))
        x = torch.where(reset, nx, a * nx + (1.0 - a) * ax)
        y = torch.where(reset, ny, a * ny + (1.0 - a) * ay)
        ax, ay = torch.where(reset, x, ax), torch.where(reset, y, ay)
        count = torch.where(reset, 0.0, count + 1.0)
        reset = torch.zeros_like(reset)
        since = since + 1.0
        if (it + 1) % CHECK_EVERY:
            continue
        measure = (omega * dx.square().sum(0) + dy.square().sum(0) / omega).sqrt()
        at_restart = torch.where(at_restart.isfinite(), at_restart, measure)
        go = ((measure <= 0.2 * at_restart) | ((measure <= 0.8 * at_restart) & (measure > last))
              | (since >= 0.36 * (it + 1)))
        last = torch.where(go, math.inf, measure)
        delta_x, delta_y = (x - xr).norm(dim=0), (y - yr).norm(dim=0)
        move = go & seen & (delta_x > 1e-12) & (delta_y > 1e-12)
        error = torch.where(move, omega * delta_x / delta_y, 1.0).log()
        omega = torch.where(move, (omega.log() - 0.5 * error - 0.3 * (error - previous)).exp(),
                            omega)
        previous = torch.where(move, error, previous)
        seen = seen | go
        at_restart = torch.where(go, measure, at_restart)
        since = torch.where(go, 0.0, since)
        reset = go
        xr, yr = torch.where(go, x, xr), torch.where(go, y, yr)
    x, y = x * d2, y * d1
    objective = lp.objective_scale * (c * x).sum(0) + lp.objective_offset
    return x.T.cpu().numpy(), y.T.cpu().numpy(), objective.cpu().numpy()


def _exact_unrolled(lp, c, q, lower, upper, price, iterations, period):
    s = _Scaled(lp.k)
    c, q, lower, upper, price = (_t(a).T.contiguous() for a in (c, q, lower, upper, price))
    d1, d2 = s.d1[:, None], s.d2[:, None]
    cs, qs, lo, hi = c * d2, q * d1, lower / d2, upper / d2
    eta = 0.9 / s.norm
    omega = cs.norm(dim=0) / qs.norm(dim=0)
    tau, sigma = eta / omega, eta * omega
    cone = (torch.arange(s.m, device=cs.device) >= lp.num_equalities)[:, None]
    x = torch.zeros_like(cs)
    x = torch.where(x < lo, torch.where(lo.isfinite(), lo, 0.0), x)
    x = torch.where(x > hi, torch.where(hi.isfinite(), hi, 0.0), x)
    y = torch.zeros_like(qs)
    ax, ay = torch.zeros_like(x), torch.zeros_like(y)
    masks = []
    for t in range(iterations):
        a = (t % period) / (t % period + 1.0)
        u = x - tau * (cs - s.kt @ y)
        inside = (u > lo) & (u < hi)
        bar = 2.0 * torch.minimum(torch.maximum(u, lo), hi) - x
        w = y + sigma * (qs - s.k @ bar)
        live = ~cone | (w > 0)
        ny = 2.0 * torch.where(cone, w.clamp_min(0.0), w) - y
        masks.append((inside, live))
        if t % period == 0:
            x, y, ax, ay = bar, ny, bar, ny
        else:
            x, y = a * bar + (1.0 - a) * ax, a * ny + (1.0 - a) * ay
    xh, yh = d2 * price, torch.zeros_like(y)
    axh, ayh = torch.zeros_like(xh), torch.zeros_like(yh)
    gc, gq = torch.zeros_like(xh), torch.zeros_like(yh)
    for t in range(iterations - 1, -1, -1):
        a = (t % period) / (t % period + 1.0)
        inside, live = masks.pop()
        if t % period == 0:
            ny, nx = yh + ayh, xh + axh
            axh, ayh = torch.zeros_like(xh), torch.zeros_like(yh)
        else:
            ny, nx = a * yh, a * xh
            axh, ayh = axh + (1.0 - a) * xh, ayh + (1.0 - a) * yh
        sh = torch.where(live, 2.0 * ny, 0.0)
        gq += sigma * sh
        bh = -(s.kt @ (sigma * sh))
        uh = torch.where(inside, 2.0 * nx + 2.0 * bh, 0.0)
        gc -= tau * uh
        xh = -nx - bh + uh
        yh = -ny + sh + tau * (s.k @ uh)
    return [a.T.cpu().numpy() for a in (d2 * x, d1 * y, d2 * gc, d1 * gq)]


def _rows(*vectors):
    return tuple(np.asarray(v)[None, :] for v in vectors)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("seam", "seam_check"):
        lp, v = _seam_vectors(case, seed)
        k = lp.k
        rows_of = np.repeat(np.arange(k.rows), np.diff(k.start))

        def mul(x):
            return np.bincount(rows_of, weights=k.value * x[k.index], minlength=k.rows)

        def mul_t(y):
            return np.bincount(k.index, weights=k.value * y[rows_of], minlength=k.cols)

        if kind == "seam_check":
            kx, kty = mul(v["x"]), mul_t(v["y"])
            slack = kx / v["row_scale"] - lp.q
            reduced = lp.c - kty / v["col_scale"]
            # Every column is boxed, so its bounds absorb any reduced cost.
            bound = np.where(reduced > 0, reduced * lp.lower, reduced * lp.upper).sum()
            return [kx, kty, np.array([
                np.square(slack).sum(), np.abs(slack).max(),
                (lp.q * v["row_scale"] * v["y"]).sum(), 0.0, 0.0, bound,
                (lp.c * v["col_scale"] * v["x"]).sum()])]
        step = np.clip(v["x"] - TAU * (lp.c - mul_t(v["y"])), lp.lower, lp.upper)
        dx = step - v["x"]
        bar = step + dx
        kx_bar = mul(bar)
        dy = SIGMA * (lp.q - kx_bar)
        k_dx = 0.5 * (kx_bar - v["kx"])
        h = HALPERN
        return [h * bar + (1 - h) * v["anchor"], dx, bar,
                h * (v["y"] + dy + GAMMA * dy) + (1 - h) * v["anchor_y"], dy,
                h * (0.5 * (kx_bar + v["kx"]) + GAMMA * k_dx) + (1 - h) * v["anchor_kx"], k_dx]
    if kind == "solve":
        # The planted dual and objective; the optimal face has more than one x.
        lp, x0, y0 = _sparse_lp(case["lp"], case["rows"], seed)
        return [None, y0, float(lp.c @ x0)]
    if kind == "resolve":
        lp, c, q = _resolve_inputs(case, seed)
        x, y, obj = _exact_solve(lp, *_rows(c, q, lp.lower, lp.upper), case["iterations"])
        return [x[0], y[0], float(obj[0])]
    if kind == "run":
        lp = _sparse_lp(case["lp"], case["rows"], seed)[0]
        x, y, obj = _exact_solve(lp, *_rows(lp.c, lp.q, lp.lower, lp.upper), case["iterations"])
        return [x[0], y[0], float(obj[0])]
    if kind == "stack":
        lp, c, q, lower, upper = _stack_inputs(case, seed)
        x, y, obj = _exact_solve(lp, c, q, lower, upper, case["iterations"])
        return [x, y, obj]
    if kind == "packed":
        out = []
        for lp in _packed_inputs(case, seed):
            x, y, obj = _exact_solve(lp, *_rows(lp.c, lp.q, lp.lower, lp.upper),
                                     case["iterations"])
            out.append([x[0], y[0], float(obj[0])])
        return out
    lp, c, q, lower, upper = _stack_inputs(case, seed)
    price = c * (1.0 + 0.05 * _rng(seed, 6).standard_normal(c.shape))
    return _exact_unrolled(lp, c, q, lower, upper, price, case["iterations"],
                           case["checkpoint"])
