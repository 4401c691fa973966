"""A resident solve holds every SM's shared memory while a launch lasts, so that a
kernel of another stream which needs shared memory waits for its end: no launch
takes more than 256 iterations, whatever the limit, and the solve is the same as
in one piece (the iterates are checked in test_gpu_resident.py)."""

import pytest

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
