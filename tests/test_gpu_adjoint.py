"""The LP adjoint (vk_lp_adjoint) on the GPU.

Pins (the reference has no differentiation):
* the CPU FP64 active-set KKT gradient (oracle/adjoint.py) at the same
  (x, y): the device LSQR must reproduce the sparse-LU / LSQR answer to 1e-8;
* end to end from the device's own solves (batched, float64, 1e-9 relative
  KKT) against the oracle gradient at HiGHS's optimum: <= 1e-4 relative;
* central finite differences (h = 1e-6, HiGHS re-solves) along random
  directions: <= 1e-4 relative;
* a thin torch.autograd.Function over the C ABI (this harness only): the
  gradients autograd returns equal the oracle's.
"""

import numpy as np
import pytest
import torch

import vikalp_b200 as vk
from oracle import adjoint as oadj
from vikalp_b200 import synthetic

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-4


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.fixture(scope="module")
def lps():
    return [synthetic.lp_uniform(200, 400, 8, seed=31 + s) for s in range(6)]


@pytest.fixture(scope="module")
def highs(lps):
    return [oadj.highs_solve(inst) for inst in lps]


def test_lsqr_matches_oracle_at_the_same_point(lps, highs):
    rng = np.random.default_rng(5)
    gs = [rng.standard_normal(i.n) for i in lps]
    got = vk.lp_adjoint(lps, [h[0] for h in highs], [h[1] for h in highs], gs, active_tolerance=1e-8)
    for inst, (x, y), g, r in zip(lps, highs, gs, got):
        want = oadj.kkt_gradient(inst, x, y, g, tol=1e-8)
        assert r["status"] == "Optimal"
        assert r["rows_active"] == want["rows_active"] and r["cols_free"] == want["cols_free"]
        for k in ("b", "A"):
            assert rel(r[k], want[k]) <= 1e-8, (k, rel(r[k], want[k]))
        assert np.all(r["c"] == 0.0)


@pytest.mark.parametrize("w_obj", [0.0, 1.0])
def test_end_to_end_against_oracle_and_fd(lps, highs, w_obj):
    sols = vk.batch_solve(lps, iteration_limit=500000, relative_tolerance=1e-9)
    assert all(s["status"] == "Optimal" for s in sols)
    rng = np.random.default_rng(11)
    gs = [rng.standard_normal(i.n) for i in lps]
    got = vk.lp_adjoint(lps, [s["x"] for s in sols], [s["y"] for s in sols], gs, dL_dobj=w_obj)
    for b, (inst, (x, y), g, r) in enumerate(zip(lps, highs, gs, got)):
        want = oadj.kkt_gradient(inst, x, y, g, w_obj=w_obj)
        for k in ("b", "A", "c"):
            if np.linalg.norm(want[k]) > 0:
                assert rel(r[k], want[k]) <= GRAD_TOL, (b, k, rel(r[k], want[k]))
        if b < 2:  # finite differences (two HiGHS re-solves per direction)
            for k, size in (("b", inst.m), ("A", inst.nnz), ("c", inst.n)):
                d = rng.standard_normal(size)
                fd = oadj.fd_directional(inst, g, {k: d}, w_obj=w_obj)
                an = float(r[k] @ d)
                assert abs(fd - an) <= GRAD_TOL * max(1.0, abs(fd)), (b, k, fd, an)


class LPLayer(torch.autograd.Function):
    """x* = argmin c'x s.t. A x <= / = b, l <= x <= u, differentiable in
    (c, b, A values) through vk_lp_adjoint. Test harness only."""

    @staticmethod
    def forward(ctx, c, b, avals, inst):
        m = synthetic.Instance(**{**inst.__dict__})
        m.c = c.detach().double().numpy()
        eq = np.isfinite(inst.row_lower) & (inst.row_lower == inst.row_upper)
        m.row_upper = b.detach().double().numpy().copy()
        m.row_lower = np.where(eq, m.row_upper, inst.row_lower)
        m.values = avals.detach().double().numpy()
        s = vk.batch_solve([m], iteration_limit=500000, relative_tolerance=1e-9)[0]
        ctx.model, ctx.x, ctx.y = m, s["x"], s["y"]
        return torch.from_numpy(s["x"].copy())

    @staticmethod
    def backward(ctx, gx):
        r = vk.lp_adjoint([ctx.model], [ctx.x], [ctx.y], [gx.double().numpy()])[0]
        return torch.from_numpy(r["c"]), torch.from_numpy(r["b"]), torch.from_numpy(r["A"]), None


def test_autograd_function(lps, highs):
    inst = lps[0]
    c = torch.tensor(inst.c, requires_grad=True)
    b = torch.tensor(inst.row_upper, requires_grad=True)
    a = torch.tensor(inst.values, requires_grad=True)
    g = torch.from_numpy(np.random.default_rng(2).standard_normal(inst.n))
    x = LPLayer.apply(c, b, a, inst)
    (x * g).sum().backward()
    want = oadj.kkt_gradient(inst, *highs[0], g.numpy())
    assert rel(b.grad.numpy(), want["b"]) <= GRAD_TOL
    assert rel(a.grad.numpy(), want["A"]) <= GRAD_TOL
    assert torch.all(c.grad == 0)


def _planted(m, n, free, per_col, seed):
    """A model with a known optimum: every row active, `free` columns inside
    their bounds (fewer than rows, so the adjoint system is consistent)."""
    rng = np.random.default_rng(seed)
    inst = synthetic.lp_uniform(m, n, per_col, seed=seed)
    x = np.where(np.arange(n) < free, rng.uniform(1, 9, n), 0.0)
    ax = synthetic.csr_matvec(inst.row_offsets, inst.col_idx, inst.values, x)
    inst.row_lower, inst.row_upper = np.full(m, -np.inf), ax
    return inst, x, rng.uniform(0, 1, m)


def test_instances_that_fit_one_sm_and_one_that_does_not():
    # the last instance's kept nonzeros (2,000 free columns x 8) exceed one
    # SM's shared memory; the others take one CTA each: a single row, no free
    # column, one free column, a zero gradient, an odd size. Against the dense
    # minimum-norm solution; 1e-8 as at the oracle's point (LSQR to 1e-12,
    # condition numbers below 1e3).
    shapes = [(1, 3, 1, 1), (40, 60, 0, 3), (40, 60, 1, 3), (333, 701, 200, 7), (333, 701, 200, 7), (2500, 3500, 2000, 8)]
    models = [_planted(*s, seed=50 + k) for k, s in enumerate(shapes)]
    rng = np.random.default_rng(9)
    gs = [rng.standard_normal(i.n) for i, _, _ in models]
    gs[3][:] = 0.0
    got = vk.lp_adjoint([t[0] for t in models], [t[1] for t in models], [t[2] for t in models], gs, 0.5,
                        solve_tolerance=1e-12)
    for (inst, x, y), (m, n, free, _), g, r in zip(models, shapes, gs, got):
        assert r["status"] == "Optimal" and r["rows_active"] == m and r["cols_free"] == free
        M = inst.dense()[:, :free].T
        keep = np.abs(M).sum(axis=1) > 0
        w = M[keep].T @ np.linalg.solve(M[keep] @ M[keep].T, g[:free][keep]) if keep.any() else np.zeros(m)
        want = {"b": w - 0.5 * y, "c": 0.5 * x}
        rows = np.repeat(np.arange(m), np.diff(inst.row_offsets))
        want["A"] = -want["b"][rows] * x[inst.col_idx]
        for k in want:
            if np.linalg.norm(want[k]) > 0:
                assert rel(r[k], want[k]) <= 1e-8, (m, k, rel(r[k], want[k]))


def test_gradients_do_not_depend_on_the_other_instances():
    # a wide instance with few kept nonzeros (180 KB of vectors) and a narrow one
    # with many (6,000, 120 KB): each fits one SM, one layout for both would not.
    # The same bits alone, in either order and beside an instance that does not fit
    # (2,000 x 8 kept); the reference point of both is the test above.
    shapes = [(200, 15_000, 50, 3), (1000, 1500, 750, 8), (2500, 3500, 2000, 8)]
    wide, narrow, large = [_planted(*s, seed=70 + k) for k, s in enumerate(shapes)]
    rng = np.random.default_rng(3)
    g = {id(i): rng.standard_normal(i[0].n) for i in (wide, narrow, large)}

    def run(models):
        return vk.lp_adjoint([t[0] for t in models], [t[1] for t in models], [t[2] for t in models],
                             [g[id(t)] for t in models], 0.5, solve_tolerance=1e-12)

    alone = {id(t): run([t])[0] for t in (wide, narrow)}
    for models in ([wide, narrow], [narrow, wide], [wide, large, narrow]):
        for t, r in zip(models, run(models)):
            if t is large:
                continue
            want = alone[id(t)]
            assert r["status"] == want["status"] == "Optimal" and r["iterations"] == want["iterations"]
            for k in ("b", "A"):
                assert np.array_equal(r[k], want[k]), (t[0].n, [u[0].n for u in models], k)
