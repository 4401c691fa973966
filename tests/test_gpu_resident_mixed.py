"""Float32 iterations in the shared memory of one cluster or of the GPU against
the sparse passes (a pinned variant keeps a model on them), at the edges of
test_gpu_resident.py, at the float32 cluster's own limit and for the index types
that only float32, or only a QP, reaches; and the float64 QP with 16-bit indices
against the restatement.

A mixed solve with tolerance 0 runs its limit in float32 and one check interval
in float64, from the float32 state. Within five checks every restart falls on a
fixed check, so that both paths take the same steps and differ by the order of
the float32 sums alone. The iteration is nonexpansive: each step adds at most
the rounding of a row's sum, about sqrt(900) * 2^-24 of the largest value for the
longest row, so 300 steps stay below 300 * 30 * 6e-8 = 5e-4; the line is 1e-3."""

import numpy as np
import pytest
import scipy.sparse as sp

import vikalp_b200 as vk
from oracle import halpern
from test_gpu_resident import _ragged, _wide
from vikalp_b200 import synthetic

pytestmark = pytest.mark.gpu

MODELS = {
    "fewer_rows_than_ctas": lambda: synthetic.lp_uniform(5, 4000, 2, seed=2),
    "ragged": _ragged,
    # m + n = 8,192: the largest float32 LP of the cluster kernel, and past it
    "cluster_largest": lambda: synthetic.lp_uniform(2600, 5592, 6, seed=12),
    "cluster_past": lambda: synthetic.lp_uniform(2600, 5593, 6, seed=12),
    "wide_indices": lambda: synthetic.lp_uniform(3000, 70001, 3, seed=4),
    "widest_packed": lambda: _wide(1 << 19),
    "past_packed": lambda: _wide((1 << 19) + 1),
    # shares of 9,800 nonzeros: past a packed word's 8,192 places, 16-bit indices fit
    "long_rows_16_bit": lambda: synthetic.lp_uniform(4000, 8000, 176, seed=13),
    "qp": lambda: synthetic.qp_sparse(700, 2001, 5, seed=9),
    # shares of 8,290 nonzeros, the same
    "qp_16_bit": lambda: synthetic.qp_sparse(4000, 8000, 148, b_rows=74_000, seed=10),
    # over 2^19 columns: 32-bit indices
    "qp_32_bit": lambda: _wide_qp((1 << 19) + 1),
}


def _wide_qp(n):
    """_wide with a diagonal Q of every 7th column."""
    inst = _wide(n)
    on = np.arange(0, n, 7)
    q = sp.csr_matrix((np.random.default_rng(16).uniform(0.1, 1.0, on.size), (on, on)), shape=(n, n))
    inst.q_row_offsets, inst.q_col_idx = q.indptr.astype(np.int64), q.indices.astype(np.int64)
    inst.q_values, inst.q_nnz = q.data, int(q.nnz)
    return inst


@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("check_every,iterations", [(64, 256), (100, 300)])
def test_float32_iterations_match_the_passes(monkeypatch, name, check_every, iterations):
    inst = MODELS[name]()
    opts = dict(algorithm="halpern", precision="mixed", iteration_limit=iterations, relative_tolerance=0.0,
                check_every=check_every)
    got = vk.solve(inst, **opts)
    monkeypatch.setenv("VIKALP_B200_VARIANT", "0")
    want = vk.solve(inst, **opts)
    assert got["fp32_iterations"] == want["fp32_iterations"] == iterations
    assert got["iterations"] == want["iterations"] == iterations + check_every
    assert got["restarts"] == want["restarts"]
    # two launches an iteration there, one a check here
    assert got["kernel_launches"] + iterations < want["kernel_launches"]
    for k in ("x", "y"):
        assert np.max(np.abs(got[k] - want[k])) <= 1e-3 * (1.0 + np.abs(want[k]).max()), k


def test_float64_qp_with_16_bit_indices_matches_restatement():
    # shares of 6,100 nonzeros of A and A' and 2,360 of Q: 228 KB with packed words,
    # 199 KB with 16-bit indices, of 225 KB. (More than 2^19 columns of a float64 QP
    # do not fit, so that none takes 32-bit indices.)
    inst = synthetic.qp_sparse(4000, 8000, 109, b_rows=26_300, seed=11)
    want = halpern.solve(inst, tol=0.0, iteration_limit=192, check_every=64)
    got = vk.solve(inst, algorithm="halpern", iteration_limit=192, relative_tolerance=0.0, check_every=64)
    assert got["iterations"] == want["iterations"] == 192 and got["restarts"] == want["restarts"]
    assert got["kernel_launches"] < 192  # resident: one launch
    for k in ("x", "y"):
        assert np.max(np.abs(got[k] - want[k])) <= 1e-8 * (1.0 + np.abs(want[k]).max()), k
