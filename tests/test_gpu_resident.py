"""Solves whose model iterates in the shared memory of one cluster or of the GPU
(vk_halpern_cluster.cuh, vk_resident.cuh) against the NumPy restatement, at
the shapes where their partition, their lanes per row and their launches have
edges: one row and column, empty rows and columns, rows long enough for a whole
warp beside single entries, indices over 16 bits and over the packed 19, more
CTAs than rows, several launches, check intervals that are no multiple of its
tables. Only the order of the sums differs from the
restatement: 1e-8 relative after a few hundred iterations, as for the passes."""

import types

import numpy as np
import pytest
import scipy.sparse as sp

import vikalp_b200 as vk
from oracle import halpern
from vikalp_b200 import synthetic

pytestmark = pytest.mark.gpu


def _model(A, seed, lo=0.0, hi=10.0):
    """An LP around a feasible point with the CSR matrix A."""
    A = sp.csr_matrix(A)
    A.sort_indices()
    m, n = A.shape
    rng = np.random.default_rng(seed)
    x0 = rng.uniform(lo, hi, n)
    ax = A @ x0
    rl, ru = ax.copy(), ax.copy()
    rl[1::2] = -np.inf
    ru[1::2] += rng.uniform(0, 1, ru[1::2].shape)
    return types.SimpleNamespace(m=m, n=n, row_offsets=A.indptr.astype(np.int64), col_idx=A.indices.astype(np.int64),
                                 values=A.data.astype(np.float64), c=rng.uniform(-1, 1, n), var_lower=np.full(n, lo),
                                 var_upper=np.full(n, hi), row_lower=rl, row_upper=ru, q_row_offsets=None,
                                 q_col_idx=None, q_values=None, q_nnz=0, objective_offset=0.0)


def _edge(n_extra):
    """m + n = 4,096 (the largest float64 LP of the cluster kernel) and past it."""
    return synthetic.lp_uniform(1300, 2796 + n_extra, 6, seed=12)


def _ragged():
    """400 x 900: one full row, one full column, empty rows and columns, single entries."""
    A = sp.random(400, 900, density=0.004, random_state=5, data_rvs=np.random.default_rng(5).standard_normal).tolil()
    rng = np.random.default_rng(6)
    A[3, :] = rng.standard_normal(900)
    A[:, 11] = rng.standard_normal((400, 1))
    A[20:30, :] = 0
    A[:, 50:60] = 0
    return _model(A.tocsr(), 7)


def _wide(n):
    """2,000 rows, entries in every 13th column and in the first and last of n, the rest empty."""
    rng = np.random.default_rng(14)
    cols = np.r_[0, np.arange(1, n - 1, 13), n - 1]
    return _model(sp.csr_matrix((rng.standard_normal(len(cols)), (rng.integers(0, 2000, len(cols)), cols)), (2000, n)), 15)


MODELS = {
    "one_by_one": lambda: _model(np.array([[1.5]]), 1),
    "fewer_rows_than_ctas": lambda: synthetic.lp_uniform(5, 4000, 2, seed=2),
    "ragged": _ragged,
    "cluster_largest": lambda: _edge(0),
    "cluster_past": lambda: _edge(1),
    "wide_indices": lambda: synthetic.lp_uniform(3000, 70001, 3, seed=4),
    "skewed": lambda: synthetic.lp_powerlaw(2001, 4003, 40_000, seed=8),
    # 19 bits hold the columns of a packed index: the last LP that they do, the
    # first that they don't, and shares that only fit with 16-bit indices
    "widest_packed": lambda: _wide(1 << 19),
    "past_packed": lambda: _wide((1 << 19) + 1),
    "long_rows_16_bit": lambda: synthetic.lp_uniform(4000, 8000, 138, seed=13),
    "qp": lambda: synthetic.qp_sparse(700, 2001, 5, seed=9),
}


@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("check_every,iterations", [(64, 192), (100, 300)])
def test_iterates_match_restatement(name, check_every, iterations):
    inst = MODELS[name]()
    want = halpern.solve(inst, tol=0.0, iteration_limit=iterations, check_every=check_every)
    got = vk.solve(inst, algorithm="halpern", iteration_limit=iterations, relative_tolerance=0.0,
                   check_every=check_every)
    assert got["iterations"] == want["iterations"] == iterations
    assert got["restarts"] == want["restarts"]
    for k in ("x", "y"):
        assert np.max(np.abs(got[k] - want[k])) <= 1e-8 * (1.0 + np.abs(want[k]).max()), k


def test_several_launches_and_repeated_solves():
    # over 1,024 iterations a solve takes more than one launch; a second solve
    # of the handle starts again from the same state
    inst = synthetic.lp_uniform(600, 1500, 6, seed=77)
    want = halpern.solve(inst, tol=0.0, iteration_limit=1216, check_every=64)
    with vk.Pdhg(inst, algorithm="halpern", relative_tolerance=0.0, iteration_limit=1216) as h:
        runs = [h.solve() for _ in range(2)]
    for r in runs:
        assert r["iterations"] == 1216 and r["restarts"] == want["restarts"]
        for k in ("x", "y"):
            assert np.max(np.abs(r[k] - want[k])) <= 1e-8 * (1.0 + np.abs(want[k]).max()), k
    assert np.array_equal(runs[0]["x"], runs[1]["x"]) and np.array_equal(runs[0]["y"], runs[1]["y"])


@pytest.mark.parametrize("name", [k for k in MODELS if k != "qp"])
@pytest.mark.parametrize("iterations", [1, 51, 52, 157, 1030])
def test_reference_scheme_matches_oracle(oracle, name, iterations):
    # FAST order: the oracle's iterates to 1e-9 through the step rule's
    # iterations (51, 101, ...) and a second launch (over 1,024)
    inst = MODELS[name]()
    tol = dict(primal_tolerance=0.0, dual_tolerance=0.0)
    want = oracle.pdhg_solve(inst, iteration_limit=iterations, **tol)
    got = vk.solve(inst, algorithm="reference", iteration_limit=iterations, **tol)
    if want["iterations"] == iterations:
        assert got["iterations"] == iterations
    else:  # one row and column: the metric reaches exactly 0, at an iteration that rounding decides
        assert name == "one_by_one" and got["last_metric"] == 0.0
    for k in ("x", "y"):
        assert np.max(np.abs(got[k] - want[k]), initial=0.0) <= 1e-9 * (1.0 + np.abs(want[k]).max()), k
