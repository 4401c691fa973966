"""A resident solve holds every SM's shared memory while a launch lasts, so that a
kernel of another stream which needs shared memory waits for its end: no launch
takes more than 256 iterations, whatever the limit, and the solve is the same as
in one piece (the iterates are checked in test_gpu_resident.py). The adjoint's
one-CTA instances take at most 1,024 iterations a launch."""

import threading
import types

import numpy as np
import pytest
import torch

import vikalp_b200 as vk
from vikalp_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lp():
    return synthetic.lp_uniform(2000, 5000, 8, seed=1)  # over 32 KB of vectors: the whole GPU


@pytest.mark.parametrize("iterations", [64, 256, 320, 1024, 1088, 2560])
def test_halpern(lp, iterations):
    r = vk.solve(lp, algorithm="halpern", iteration_limit=iterations, relative_tolerance=0.0)
    assert r["iterations"] == iterations and r["kernel_launches"] == -(-iterations // 256)


@pytest.mark.parametrize("iterations", [1, 255, 256, 600, 1024, 2500])
def test_reference(lp, iterations):
    # the stop is taken at the start of the iteration after the last
    r = vk.solve(lp, algorithm="reference", iteration_limit=iterations, primal_tolerance=0.0, dual_tolerance=0.0)
    assert r["iterations"] == iterations and r["kernel_launches"] == iterations // 256 + 1


def test_a_cluster_leaves_the_other_sms_free_and_is_not_split():
    inst = synthetic.lp_uniform(300, 800, 5, seed=1)
    r = vk.solve(inst, algorithm="halpern", iteration_limit=1024, relative_tolerance=0.0)
    assert r["iterations"] == 1024 and r["kernel_launches"] == 1


def _scaled(m, n, density, decades, seed):
    """A model at an interior point of its n columns with m active rows over so many
    decades of scale (LSQR needs many iterations): instance, point, gradient, A."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, n)) * (rng.random((m, n)) < density)
    A *= 10.0 ** rng.uniform(-decades / 2, decades / 2, (m, 1))
    rows, cols = np.nonzero(A)
    off = np.r_[0, np.cumsum(np.bincount(rows, minlength=m))].astype(np.int64)
    x = rng.uniform(1.0, 9.0, n)
    ax = A @ x
    inst = types.SimpleNamespace(m=m, n=n, row_offsets=off, col_idx=cols.astype(np.int64), values=A[rows, cols],
                                 c=np.zeros(n), var_lower=np.zeros(n), var_upper=np.full(n, 10.0), row_lower=ax,
                                 row_upper=ax, q_row_offsets=None, q_col_idx=None, q_values=None, q_nnz=0,
                                 objective_offset=0.0)
    return inst, x, rng.standard_normal(n), A


def test_adjoint_lets_other_streams_in():
    # 160 instances, one on every SM, for 100,000 iterations: about 0.4 s on the device
    inst, x, g, _ = _scaled(200, 150, 0.2, 8, seed=1)
    count, limit = 160, 100_000
    a = torch.randn(2048, 2048, device="cuda", dtype=torch.bfloat16)
    stream = torch.cuda.Stream()
    waits, out = [], []
    stop = threading.Event()

    def products():
        with torch.cuda.stream(stream):
            while not stop.is_set():
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record()
                torch.mm(a, a)
                e[1].record()
                e[1].synchronize()
                waits.append(e[0].elapsed_time(e[1]))

    with torch.cuda.stream(stream):
        torch.mm(a, a)
    stream.synchronize()
    t = threading.Thread(target=products)
    t.start()
    try:
        out = vk.lp_adjoint([inst] * count, [x] * count, [np.zeros(200)] * count, [g] * count, solve_tolerance=1e-300,
                            iteration_limit=limit)
    finally:
        stop.set()
        t.join()
    for r in out:
        assert r["status"] == "IterationLimit" and r["iterations"] == limit
        assert np.array_equal(r["b"], out[0]["b"])
    # a launch of 1,024 iterations takes 1% of the call's; in one launch a product waits for all
    assert max(waits) < 100.0, max(waits)


def test_adjoint_over_several_launches_converges():
    # 60 equations, 40 unknowns over four decades: some 7,000 iterations, seven launches,
    # until the residual of the normal equations vanishes. Against the dense solution:
    # condition 8e3 squared (an inconsistent system) times 2^-53 is 7e-9; the line is 4e-8.
    inst, x, g, A = _scaled(40, 60, 0.2, 4, seed=1)
    r = vk.lp_adjoint([inst], [x], [np.zeros(40)], [g], solve_tolerance=1e-300, iteration_limit=100_000)[0]
    want = np.linalg.lstsq(A.T, g, rcond=1e-14)[0]
    assert r["status"] == "Optimal" and r["iterations"] > 2048
    assert np.linalg.norm(r["b"] - want) <= 4e-8 * np.linalg.norm(want)
    cut = vk.lp_adjoint([inst], [x], [np.zeros(40)], [g], solve_tolerance=1e-300, iteration_limit=1025)[0]
    assert cut["status"] == "IterationLimit" and cut["iterations"] == 1025
