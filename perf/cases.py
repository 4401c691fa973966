"""The calls this library's speed is judged by: its public entry points over the
sizes, structures and options its users run.

A case is one of five kinds of call, each made as a user's program makes it:

* ``solve``     -- a model resident on the GPU (``Pdhg``) is solved once more for new
                   variable bounds, from a warm start where there is one;
* ``nodes``     -- branch-and-bound relaxations of one LP in one call
                   (``batch_solve_shared``), set-up included;
* ``lps``       -- independent LPs of uneven size in one call (``batch_solve``),
                   set-up included;
* ``adjoint``   -- gradients of solved LPs (``lp_adjoint``), set-up included;
* ``products``  -- A x and A'y of a resident operator on device vectors (``SpMat``).

Solves run to their iteration limit (the relative tolerance is 0): the budget a
node of a search tree gets, and the same number of iterations in every run.
Models are drawn on the GPU from the seed alone, with the distributions of
``vikalp_b200.synthetic``: N(0,1) values on ``per_col`` uniform rows per column, or
Zipf(1.5) column counts with values over six decades; a box [0, 10]; half of the
rows equations and half inequalities through a feasible point.
"""

from __future__ import annotations

import types

import numpy as np
import torch

import vikalp_b200 as vk

INF = float("inf")
CHECK = 64  # iterations between the Halpern scheme's checks (the library's default)


def listed() -> list[dict]:
    """The cases, from the smallest call to the largest."""
    return [
        # a plain product of a small operator, float32: one call is a few microseconds of work
        dict(name="products_small_fp32", kind="products", structure="uniform", m=20_011, n=40_001, per_col=6,
             precision="mixed"),
        # one node of a small search tree, warm-started: the smallest solve, all latency
        dict(name="node_tiny", kind="solve", scheme="halpern", structure="uniform", m=300, n=800, per_col=5,
             iterations=320, precision="fp64", warm=True),
        # the small LP in the reference's own scheme (the router's default)
        dict(name="lp_small_reference", kind="solve", scheme="reference", structure="uniform", m=2_000, n=5_000,
             per_col=8, iterations=600, precision="fp64", warm=False),
        # the small LP in the restarted Halpern scheme
        dict(name="lp_small_halpern", kind="solve", scheme="halpern", structure="uniform", m=2_000, n=5_000,
             per_col=8, iterations=1_280, precision="fp64", warm=False),
        # the root relaxation of the batched workload's LP
        dict(name="lp_medium_halpern", kind="solve", scheme="halpern", structure="uniform", m=50_000, n=100_000,
             per_col=6, iterations=640, precision="fp64", warm=False),
        # an LP of odd sizes in mixed precision (float32 iterations, a float64 finish)
        dict(name="lp_medium_mixed", kind="solve", scheme="halpern", structure="uniform", m=99_999, n=210_001,
             per_col=8, iterations=256, precision="mixed", warm=True),
        # the large power-law LP in the reference's scheme: the benchmark's workload
        dict(name="lp_large_reference", kind="solve", scheme="reference", structure="powerlaw", m=1_000_000,
             n=2_000_000, per_col=10, iterations=200, precision="fp64", warm=False),
        # a convex QP: the same passes plus one over Q
        dict(name="qp_halpern", kind="solve", scheme="halpern", structure="qp", m=40_000, n=100_000, per_col=6,
             iterations=512, precision="fp64", warm=False),
        # nodes of one LP solved together
        dict(name="nodes_shared", kind="nodes", structure="uniform", m=10_000, n=20_000, per_col=6, count=128,
             iterations=960, precision="fp64"),
        # independent LPs solved together, sizes log-uniform from 500 rows up
        dict(name="lps_uneven", kind="lps", structure="uniform", m=8_000, per_col=8, count=48, iterations=1_280,
             precision="fp64"),
        # gradients of a batch of solved LPs
        dict(name="adjoint", kind="adjoint", m=1_000, n=2_000, per_col=8, count=64),
        # plain products of a large skewed operator, both directions
        dict(name="products_large_fp64", kind="products", structure="powerlaw", m=500_000, n=1_000_000, per_col=10,
             precision="fp64"),
    ]


def _size(rng, lo: int, hi: int) -> int:
    """Log-uniform on [lo, hi], odd more often than not."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(lo, min(hi, v | 1 if rng.random() < 0.6 else v))


def draw(rng) -> dict:
    """One more case of the listed ranges."""
    kind = rng.choice(["solve", "solve", "solve", "products", "nodes", "lps", "adjoint"])
    if kind == "solve":
        structure = rng.choice(["uniform", "uniform", "powerlaw", "qp"])
        m = _size(rng, *{"uniform": (300, 100_000), "powerlaw": (20_000, 400_000), "qp": (2_000, 40_000)}[structure])
        n = int(m * rng.uniform(1.5, 2.7))
        scheme = "halpern" if structure == "qp" else rng.choice(["halpern", "reference"])
        # (values over six decades: a float32 trajectory says little, so float64)
        precision = rng.choice(["fp64", "mixed"]) if scheme == "halpern" and structure != "powerlaw" else "fp64"
        # a float32 trajectory is comparable while every restart falls on a fixed check (the first five)
        iterations = 64 * rng.randint(2, 4) if precision == "mixed" else rng.choice([200, 320, 500, 640])
        return dict(kind=kind, scheme=scheme, structure=structure, m=m, n=n,
                    per_col=10 if structure == "powerlaw" else rng.randint(4, 9), iterations=iterations,
                    precision=precision, warm=rng.random() < 0.5)
    if kind == "products":
        structure = rng.choice(["uniform", "powerlaw"])
        m = _size(rng, 1_000, 500_000)
        return dict(kind=kind, structure=structure, m=m, n=int(m * rng.uniform(0.7, 2.5)), per_col=rng.randint(4, 10),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "nodes":
        m, precision = _size(rng, 1_000, 10_000), rng.choice(["fp64", "mixed"])
        return dict(kind=kind, structure="uniform", m=m, n=int(m * rng.uniform(1.5, 2.2)), per_col=rng.randint(4, 8),
                    count=rng.randint(20, 140), iterations=256 if precision == "mixed" else 640, precision=precision)
    if kind == "lps":
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, structure="uniform", m=_size(rng, 1_000, 8_000), per_col=rng.randint(4, 8),
                    count=rng.randint(8, 48), iterations=256 if precision == "mixed" else 640, precision=precision)
    m = _size(rng, 300, 1_000)
    return dict(kind=kind, m=m, n=int(m * rng.uniform(1.6, 2.2)), per_col=rng.randint(6, 9), count=rng.randint(8, 64))


# ---- models ---------------------------------------------------------------------


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _row_sums(values, offsets):
    """Sums of the CSR rows, left to right (the same bits every time)."""
    return torch.segment_reduce(values, "sum", lengths=offsets.diff(), unsafe=True, initial=0.0)


def _pattern(g, m, n, degrees):
    """CSR offsets and columns: degrees[j] uniform rows for column j, repeats merged."""
    cols = torch.repeat_interleave(torch.arange(n, device="cuda"), degrees)
    rows = torch.randint(0, m, (cols.numel(),), generator=g, device="cuda")
    return _sorted_csr(rows, cols, m, n)


def _sorted_csr(rows, cols, m, n):
    key = torch.unique(rows * n + cols)
    offsets = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.bincount(key // n, minlength=m).cumsum(0)
    return offsets, key % n


def _degrees(g, structure, n, per_col):
    if structure != "powerlaw":
        return torch.full((n,), per_col, device="cuda")
    # Zipf(1.5) clamped at 2000, thinned to per_col on average, at least 1
    k = np.arange(1, 2000)
    cdf = torch.from_numpy(np.cumsum(k ** -1.5 / 2.612375348685488)).cuda()
    deg = (torch.searchsorted(cdf, _rand(g, n)) + 1).double()
    p = torch.full_like(deg, min(1.0, per_col / 67.9))  # 67.9: the clamped law's mean
    return torch.binomial(deg, p, generator=g).long().clamp_(min=1)


def _model(g, structure, m, n, per_col):
    """A model in the caller's host arrays (int64 CSR, float64)."""
    offsets, cols = _pattern(g, m, n, _degrees(g, structure, n, per_col))
    nnz = cols.numel()
    if structure == "powerlaw":
        sign = torch.where(_rand(g, nnz) < 0.5, -1.0, 1.0).double()
        values = sign * 10.0 ** (6.0 * _rand(g, nnz) - 3.0)
    else:
        values = _normal(g, nnz)
    lo, hi = (-5.0, 5.0) if structure == "qp" else (0.0, 10.0)
    x0 = lo + (hi - lo) * _rand(g, n)
    ax0 = _row_sums(values * x0[cols], offsets)
    odd = torch.arange(m, device="cuda") % 2 == 1
    inst = types.SimpleNamespace(
        m=m, n=n, row_offsets=offsets.cpu().numpy(), col_idx=cols.cpu().numpy(), values=values.cpu().numpy(),
        c=(_normal(g, n) if structure == "qp" else 2.0 * _rand(g, n) - 1.0).cpu().numpy(),
        var_lower=np.full(n, lo), var_upper=np.full(n, hi),
        row_lower=torch.where(odd, -INF, ax0).cpu().numpy(),
        row_upper=torch.where(odd, ax0 + _rand(g, m), ax0).cpu().numpy(),
        x0=x0.cpu().numpy(), q_row_offsets=None, q_col_idx=None, q_values=None, q_nnz=0, objective_offset=0.0)
    if structure == "qp":
        # Q = D + B'B, B with n/10 rows of four N(0, 1/4) entries
        nb = n // 10
        bc = torch.randint(0, n, (nb, 4), generator=g, device="cuda")
        bv = 0.5 * _normal(g, nb, 4)
        diag = torch.arange(n, device="cuda")
        key = torch.cat([(bc[:, :, None] * n + bc[:, None, :]).flatten(), diag * n + diag])
        val = torch.cat([(bv[:, :, None] * bv[:, None, :]).flatten(), 0.1 + 0.9 * _rand(g, n)])
        key, order = torch.sort(key, stable=True)
        key, counts = torch.unique_consecutive(key, return_counts=True)
        val = torch.segment_reduce(val[order], "sum", lengths=counts, unsafe=True)
        qo = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        qo[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
        inst.q_row_offsets, inst.q_col_idx, inst.q_values = qo.cpu().numpy(), (key % n).cpu().numpy(), val.cpu().numpy()
        inst.q_nnz = int(key.numel())
    return inst


def _node_bounds(inst, count, seed):
    """Bounds of `count` nodes: each tightens up to twelve variables around the feasible point."""
    rng = np.random.default_rng(seed)
    lo, hi = np.tile(inst.var_lower, (count, 1)), np.tile(inst.var_upper, (count, 1))
    for b in range(count):
        js = rng.choice(inst.n, size=int(rng.integers(1, 13)), replace=False)
        d = rng.uniform(0.0, 2.0, size=js.size)
        down = rng.integers(0, 2, size=js.size) == 1
        hi[b, js[down]] = np.clip(np.floor(inst.x0[js] + d)[down], inst.var_lower[js[down]], inst.var_upper[js[down]])
        lo[b, js[~down]] = np.clip(np.ceil(inst.x0[js] - d)[~down], inst.var_lower[js[~down]], hi[b, js[~down]])
    return lo, hi


def _solved_lp(g, m, n, per_col):
    """An LP with a known (degenerate) optimum: 4/5 of the rows active, 3/10 of
    the columns strictly inside their bounds. Returns (model, x, y, dL/dx)."""
    rows = _rand(g, n, m).topk(per_col, dim=1).indices  # distinct: every model has n * per_col nonzeros
    offsets, cols = _sorted_csr(rows.flatten(), torch.arange(n, device="cuda").repeat_interleave(per_col), m, n)
    values = _normal(g, cols.numel())
    u = _rand(g, n)
    x = torch.where(u < 0.3, 1.0 + 8.0 * _rand(g, n), torch.where(u < 0.65, 0.0, 10.0))
    ax = _row_sums(values * x[cols], offsets)
    active = _rand(g, m) < 0.8
    y = torch.where(active, _rand(g, m), 0.0)
    rows = torch.repeat_interleave(torch.arange(m, device="cuda"), offsets.diff())
    order = torch.sort(cols, stable=True).indices
    aty = torch.segment_reduce((values * y[rows])[order], "sum", lengths=torch.bincount(cols, minlength=n),
                               unsafe=True, initial=0.0)
    reduced = torch.where(u < 0.3, 0.0, torch.where(u < 0.65, 1.0, -1.0)) * _rand(g, n)
    inst = types.SimpleNamespace(
        m=m, n=n, row_offsets=offsets.cpu().numpy(), col_idx=cols.cpu().numpy(), values=values.cpu().numpy(),
        c=(reduced - aty).cpu().numpy(), var_lower=np.zeros(n), var_upper=np.full(n, 10.0),
        row_lower=np.full(m, -INF), row_upper=torch.where(active, ax, ax + 1.0).cpu().numpy(), q_col_idx=None,
        q_nnz=0, objective_offset=0.0)
    return inst, x.cpu().numpy(), y.cpu().numpy(), _normal(g, n).cpu().numpy()


def _uneven_sizes(case) -> list[int]:
    """Row counts of the independent LPs: log-spaced from 500 (or m, if smaller) to m."""
    lo = min(500, case["m"])
    return [int(lo * (case["m"] / lo) ** (b / max(1, case["count"] - 1))) for b in range(case["count"])]


def _inputs(case, seed):
    """What the call is made with, as the caller holds it."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "lps":
        return dict(lps=[_model(g, "uniform", m, 2 * m, case["per_col"]) for m in _uneven_sizes(case)])
    if kind == "adjoint":
        solved = [_solved_lp(g, case["m"], case["n"], case["per_col"]) for _ in range(case["count"])]
        return dict(zip(("lps", "x", "y", "grad"), (list(t) for t in zip(*solved))))
    inst = _model(g, case["structure"], case["m"], case["n"], case["per_col"])
    if kind == "nodes":
        lo, hi = _node_bounds(inst, case["count"], seed)
        return dict(inst=inst, lower=lo, upper=hi)
    if kind == "products":
        dt = torch.float32 if case["precision"] == "mixed" else torch.float64
        return dict(inst=inst, x=_rand(g, case["n"]).to(dt), y=_normal(g, case["m"]).to(dt))
    lo, hi = _node_bounds(inst, 1, seed)
    # warm start: the parent's point, about 0.1 away from feasible
    warm = inst.x0 + 0.1 * _normal(g, case["n"]).cpu().numpy() if case["warm"] else None
    return dict(inst=inst, lower=lo[0], upper=hi[0], warm=warm)


def _options(case) -> dict:
    if case.get("scheme") == "reference":
        return dict(algorithm="reference", iteration_limit=case["iterations"], primal_tolerance=0.0,
                    dual_tolerance=0.0)
    return dict(algorithm="halpern", precision=case["precision"], iteration_limit=case["iterations"],
                relative_tolerance=0.0)


def prepare(case, seed):
    """Inputs, and the handle a user's program keeps: a resident model or operator."""
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "solve":
        s["handle"] = vk.Pdhg(s["inst"], **_options(case))
    elif case["kind"] == "products":
        i = s["inst"]
        s["op"] = vk.SpMat(i.row_offsets, i.col_idx, i.values, i.m, i.n, case["precision"])
        s["ax"], s["aty"] = torch.empty_like(s["y"]), torch.empty_like(s["x"])
    return s


def _answer(case, results):
    """The solutions of one call; a mixed-precision answer is good to float32 and kept as float32."""
    dt = np.float32 if case["precision"] == "mixed" else np.float64
    out = {k: np.concatenate([r[k] for r in results]).astype(dt, copy=False) for k in ("x", "y")}
    if dt == np.float64:  # in float32 its terms cancel: the caller takes it from x
        out["objective"] = np.array([r["objective"] for r in results])
    out["iterations"] = np.array([r["iterations"] for r in results])
    return out


def run(state):
    """One pass."""
    case = state["case"]
    if case["kind"] == "solve":
        return _answer(case, [state["handle"].solve(state["warm"], state["lower"], state["upper"], duals=False)])
    if case["kind"] == "nodes":
        return _answer(case, vk.batch_solve_shared(state["inst"], case["count"], state["lower"], state["upper"],
                                                   **_options(case)))
    if case["kind"] == "lps":
        return _answer(case, vk.batch_solve(state["lps"], **_options(case)))
    if case["kind"] == "adjoint":
        grads = vk.lp_adjoint(state["lps"], state["x"], state["y"], state["grad"], 1.0, solve_tolerance=1e-13)
        return {k: np.concatenate([g[k] for g in grads]) for k in ("c", "b", "A")}
    stream = torch.cuda.current_stream().cuda_stream
    state["op"].apply(state["x"].data_ptr(), state["ax"].data_ptr(), False, stream)
    state["op"].apply(state["y"].data_ptr(), state["aty"].data_ptr(), True, stream)
    return {"ax": state["ax"], "aty": state["aty"]}


# ---- what a pass cannot do without ------------------------------------------------


def work(case) -> dict:
    """Bytes and operations of one pass: per iteration the matrix once for each of
    its two products and the vectors of the step once; a product its matrix,
    input and output once."""
    s = 4 if case.get("precision") == "mixed" else 8
    per = case["per_col"]
    if case["kind"] == "products":
        m, n = case["m"], case["n"]
        nnz = n * per
        return {"bytes": 2 * (nnz * (s + 4) + 4 * (m + n) // 2 + s * (m + n)), "flops": 4 * nnz}
    if case["kind"] == "adjoint":
        # at least one read of the model, x, y and dL/dx and one write of the gradients
        m, n, B = case["m"], case["n"], case["count"]
        return {"bytes": B * (n * per * (8 + 8 + 8) + 8 * (3 * n + 2 * m)), "flops": 4 * B * n * per}
    its = -(-case["iterations"] // CHECK) * CHECK if case.get("scheme") != "reference" else case["iterations"]
    if case["kind"] == "lps":
        m = sum(_uneven_sizes(case))
        n, B = 2 * m, 1
    else:
        m, n, B = case["m"], case["n"], case.get("count", 1)
    nnz = n * per
    q = n + 12 * (n // 10) if case.get("structure") == "qp" else 0
    vectors = 6 * n + 5 * m
    return {"bytes": its * ((2 * nnz + q) * (s + 4) + B * vectors * s), "flops": its * B * (4 * nnz + 2 * q + 10 * (m + n))}


# ---- 64-bit values, in plain torch ---------------------------------------------------


def _csr(offsets, cols, values, shape):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return torch.sparse_csr_tensor(t(offsets), t(cols), t(values), size=shape)


def _transposed(A):
    m, n = A.shape
    rows = torch.repeat_interleave(torch.arange(m, device="cuda"), A.crow_indices().diff())
    cols, order = torch.sort(A.col_indices(), stable=True)
    offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.bincount(cols, minlength=n).cumsum(0)
    return torch.sparse_csr_tensor(offsets, rows[order], A.values()[order], size=(n, m))


def _scaled(A, r, d):
    rows = torch.repeat_interleave(torch.arange(A.shape[0], device="cuda"), A.crow_indices().diff())
    return torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values() * r[rows] * d[A.col_indices()],
                                   size=A.shape)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _reference(inst, lo, hi, warm, iterations):
    """The reference's scheme (pdhg.cpp:61-151) for a fixed number of iterations."""
    A = _csr(inst.row_offsets, inst.col_idx, inst.values, (inst.m, inst.n))
    AT = _transposed(A)
    big = lambda M: torch.segment_reduce(M.values().abs(), "max", lengths=M.crow_indices().diff(), unsafe=True,  # noqa: E731
                                         initial=0.0)
    r, d = 1.0 / big(A).clamp(min=1.0), 1.0 / big(AT).clamp(min=1.0)
    K, KT = _scaled(A, r, d), _scaled(AT, d, r)
    total = lambda M: float(_row_sums(M.values().abs(), M.crow_indices()).max())  # noqa: E731
    top = 0.99 / max(1.0, (total(K) * total(KT)) ** 0.5)
    c, l, u = _dev(inst.c) * d, _dev(lo) / d, _dev(hi) / d
    rl, ru = _dev(inst.row_lower) * r, _dev(inst.row_upper) * r
    x = (torch.zeros_like(c) if warm is None else _dev(warm) / d).clamp(l, u)
    y = torch.zeros_like(rl)
    tau, previous, restart = top, INF, False
    aty, kx = KT @ y, K @ x
    for it in range(iterations):
        xn = (x - tau * (c + aty)).clamp(l, u)
        kxn = K @ xn
        v = y + tau * (kxn if restart else 2.0 * kxn - kx)
        y = v - tau * (v / tau).clamp(rl, ru)
        x, kx, aty, restart = xn, kxn, KT @ y, False
        if it % 50 == 0:
            metric = max(float((kx.clamp(rl, ru) - kx).abs().max()),
                         float((x - (x - (c + aty)).clamp(l, u)).abs().max()))
            if it > 0 and metric > previous * 1.25:
                tau, restart = tau * 0.5, True
            elif it > 0 and metric < previous * 0.1:
                tau = min(tau * 1.05, top)
            previous = metric
    xo, yo = x * d, y * r
    return xo, yo, iterations


def _power(mul, n, root):
    """Largest eigenvalue of a PSD operator (its root, if `root`): power iteration
    from the library's start vector, with its stopping rule."""
    h = (torch.arange(n, device="cuda") * 2654435761 + 12345) & 0xFFFFFFFF
    h ^= h >> 13
    h = (h * 2246822519) & 0xFFFFFFFF
    h ^= h >> 16
    v = 0.5 + (h & 0xFFFF).double() / 65536.0
    v /= v.norm()
    prev = 0.0
    for it in range(200):
        z = mul(v)
        nz = float(z.norm())
        est = nz ** 0.5 if root else nz
        v = z / nz
        if it > 10 and abs(est - prev) <= 1e-6 * est:
            return est
        prev = est
    return prev


def _step(knorm, lq, omega):
    """(eta, rho) per instance for primal weights omega (a vector)."""
    if lq <= 0.0:
        return torch.full_like(omega, 0.99 / knorm), torch.ones_like(omega)
    k2, b, c = knorm * knorm, lq / omega, 0.9801
    eta = 2.0 * c / (b + (b * b + 4.0 * k2 * c).sqrt())
    kappa = (1.0 - eta * eta * k2) / (eta / omega * lq)
    return eta, (0.99 * (1.0 - 1.0 / (2.0 * kappa))).clamp(max=1.0)


def _halpern(inst, lo, hi, warm, iterations, mixed):
    """The restarted reflected-Halpern scheme for a fixed number of iterations, for
    the instances (columns) of lo / hi [n, B]; a mixed solve's float64 finish is
    one more check interval."""
    m, n, B = inst.m, inst.n, lo.shape[1]
    A = _csr(inst.row_offsets, inst.col_idx, inst.values, (m, n))
    AT = _transposed(A)
    Q = _csr(inst.q_row_offsets, inst.q_col_idx, inst.q_values, (n, n)) if inst.q_nnz else None
    r, d = torch.ones(m, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    for p in range(11):
        how = "max" if p < 10 else "sum"
        red = lambda M, s, t: s * torch.segment_reduce(M.values().abs() * t[M.col_indices()], how,  # noqa: E731
                                                       lengths=M.crow_indices().diff(), unsafe=True, initial=0.0)
        rn, cn = red(A, r, d), red(AT, d, r)
        r, d = torch.where(rn > 0, r / rn.sqrt(), r), torch.where(cn > 0, d / cn.sqrt(), d)
    K, KT = _scaled(A, r, d), _scaled(AT, d, r)
    Qs = _scaled(Q, d, d) if Q is not None else None
    col = lambda a: a[:, None]  # noqa: E731
    c, l, u = col(_dev(inst.c) * d), lo / col(d), hi / col(d)
    orl, oru = _dev(inst.row_lower), _dev(inst.row_upper)
    rl, ru = col(orl * r), col(oru * r)
    b = torch.maximum(torch.where(orl.isfinite(), orl.abs(), 0.0), torch.where(oru.isfinite(), oru.abs(), 0.0))
    knorm = _power(lambda v: KT @ (K @ v), n, True)
    lq = _power(lambda v: Qs @ v, n, False) if Qs is not None else 0.0
    omega = torch.full((B,), float(c.norm()) / float((b * r).norm()), dtype=torch.float64, device="cuda")
    eta, rho = _step(knorm, lq, omega)
    x = (torch.zeros_like(l) if warm is None else warm / col(d)).clamp(l, u)
    y = torch.zeros(m, B, dtype=torch.float64, device="cuda")
    x0, y0 = x.clone(), y.clone()
    kb = torch.zeros(B, dtype=torch.float64, device="cuda")
    rr, rp = torch.full_like(omega, -1.0), torch.full_like(omega, INF)
    limit, total = -(-iterations // CHECK) * CHECK, 0
    while True:
        tau, sigma = eta / omega, eta * omega
        for it in range(CHECK):
            lam = (kb + it + 1.0) / (kb + it + 2.0)
            g = c + KT @ y if Qs is None else c + Qs @ x + KT @ y
            xh = (x - tau * g).clamp(l, u)
            v = y + sigma * (K @ (2.0 * xh - x))
            yh = v - torch.minimum(torch.maximum(v, sigma * rl), sigma * ru)
            xp, yp = x, y
            x = lam * ((1.0 + rho) * xh - rho * x) + (1.0 - lam) * x0
            y = lam * ((1.0 + rho) * yh - rho * y) + (1.0 - lam) * y0
        total += CHECK
        if total >= limit:
            if not mixed or total > limit:
                break
            continue  # the float64 finish goes on from the last state, its counter unchanged
        fp = (omega * (xh - xp).square().sum(0) + (yh - yp).square().sum(0) / omega).sqrt()
        k = kb + CHECK
        again = (rr >= 0) & ((fp <= 0.2 * rr) | ((fp <= 0.8 * rr) & (fp > rp)) | (k >= 0.2 * total))
        rr = torch.where((rr < 0) | again, fp, rr)
        rp = fp
        mx, my = (xh - x0).norm(dim=0), (yh - y0).norm(dim=0)
        w = torch.exp(0.2 * torch.log(my / mx) + 0.8 * torch.log(omega))
        omega = torch.where(again & (mx > 1e-10) & (my > 1e-10), w, omega)
        eta, rho = _step(knorm, lq, omega)
        kb = torch.where(again, 0.0, k)
        x, x0 = torch.where(again, xh, x), torch.where(again, xh, x0)
        y, y0 = torch.where(again, yh, y), torch.where(again, yh, y0)
    return xh * col(d), yh * col(r), total


def _objective(inst, x):
    """c'x + x'Qx / 2 per instance (column of x)."""
    v = _dev(inst.c) @ x
    if inst.q_nnz:
        Q = _csr(inst.q_row_offsets, inst.q_col_idx, inst.q_values, (inst.n, inst.n))
        v = v + 0.5 * (x * (Q @ x)).sum(0)
    return v


def _adjoint(inst, x, y, g):
    """Active-set adjoint with dL/dobj = 1: w = the minimum-norm least-squares solution of A_RF' w = g_F."""
    rows = np.repeat(np.arange(inst.m), np.diff(inst.row_offsets))
    dense = torch.zeros(inst.m, inst.n, dtype=torch.float64, device="cuda")
    dense[torch.from_numpy(rows).cuda(), torch.from_numpy(inst.col_idx).cuda()] = _dev(inst.values)
    ax = dense @ _dev(x)
    ru = _dev(inst.row_upper)
    active = (ax - ru).abs() <= 1e-6 * (1.0 + ru.abs())
    free = torch.from_numpy((x > 1e-6) & (x < 10.0 - 1.1e-5)).cuda()
    M = dense[active][:, free].T
    lam, V = torch.linalg.eigh(M @ M.T)
    t = V.T @ _dev(g)[free]
    w = torch.zeros(inst.m, dtype=torch.float64, device="cuda")
    w[active] = M.T @ (V @ torch.where(lam > 1e-12 * lam.max(), t / lam, 0.0))
    b = w.cpu().numpy() - y
    return {"c": x, "b": b, "A": -b[rows] * x[inst.col_idx]}


def exact(case, seed):
    """run()'s outputs in 64 bits."""
    s = _inputs(case, seed)
    if case["kind"] == "products":
        i = s["inst"]
        values = i.values.astype(np.float32).astype(np.float64) if case["precision"] == "mixed" else i.values
        A = _csr(i.row_offsets, i.col_idx, values, (i.m, i.n))
        return {"ax": A @ s["x"].double(), "aty": _transposed(A) @ s["y"].double()}
    if case["kind"] == "adjoint":
        grads = [_adjoint(*t) for t in zip(s["lps"], s["x"], s["y"], s["grad"])]
        return {k: np.concatenate([g[k] for g in grads]) for k in ("c", "b", "A")}
    mixed = case["precision"] == "mixed"
    if case["kind"] == "lps":
        done = []
        for i in s["lps"]:
            x, y, its = _halpern(i, _dev(i.var_lower)[:, None], _dev(i.var_upper)[:, None], None, case["iterations"],
                                 mixed)
            done.append((x[:, 0], y[:, 0], _objective(i, x), its))
        xs, ys, obj, its = zip(*done)
        out = {"x": torch.cat(xs), "y": torch.cat(ys), "objective": torch.cat(obj), "iterations": list(its)}
    elif case["kind"] == "nodes":
        i = s["inst"]
        x, y, its = _halpern(i, _dev(s["lower"].T), _dev(s["upper"].T), None, case["iterations"], mixed)
        out = {"x": x.T.flatten(), "y": y.T.flatten(), "objective": _objective(i, x),
               "iterations": [its] * case["count"]}
    elif case["scheme"] == "reference":
        i = s["inst"]
        x, y, its = _reference(i, s["lower"], s["upper"], s["warm"], case["iterations"])
        out = {"x": x, "y": y, "objective": _objective(i, x[:, None]), "iterations": [its]}
    else:
        i = s["inst"]
        warm = None if s["warm"] is None else _dev(s["warm"])[:, None]
        x, y, its = _halpern(i, _dev(s["lower"])[:, None], _dev(s["upper"])[:, None], warm, case["iterations"], mixed)
        out = {"x": x[:, 0], "y": y[:, 0], "objective": _objective(i, x), "iterations": [its]}
    if mixed:
        del out["objective"]
    return {k: np.array(v) if k == "iterations" else v for k, v in out.items()}
