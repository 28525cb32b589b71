"""A device allocation that fails in the middle of a call (zmpm_fail_allocation):
the call returns its error and the next one on the same context is right."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.test_gpu_binning import assert_bins_equal

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


def fail_each(lib, prepare):
    """prepare()'s scene binned with its first, second, ... allocation failing, until none is left to fail; returns the
    scenes whose pass failed."""
    failed = []
    while len(failed) < 64:
        s = prepare()
        lib.fail_allocation(len(failed) + 1)
        rc = s.lib.bin(s.ctx, None)
        lib.fail_allocation(0)
        if rc == abi.OK:
            return failed
        assert rc == abi.CUDA_ERROR
        failed.append(s)
    raise AssertionError("every pass failed")


SCENES = {
    # many pages, some shared; one page's 4000 particles (the radix way); one page (page counters would add up past P)
    "loose": lambda rng: (20 + 30 * rng.random((4000, 3))) * DX,
    "dense": lambda rng: (32.55 + 0.9 * rng.random((4000, 3))) * DX,
    "one-page": lambda rng: (32.55 + 0.9 * rng.random((900, 3))) * DX,
}


@pytest.mark.parametrize("scene", sorted(SCENES))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_binning_after_a_failed_pass(cuda_lib, oracle, scene, precision):
    x = SCENES[scene](np.random.default_rng(3)).astype(np.float32).astype(np.float64)
    o = mpm.MpmSimulation(DX, precision=precision, lib=oracle)
    o.addParticles(x, None, 1.0, 1.0)
    want = o.binParticles()

    def prepare():
        s = mpm.MpmSimulation(DX, precision=precision, grid_log2=7)
        s.addParticles(x, None, 1.0, 1.0)
        return s

    failed = fail_each(cuda_lib, prepare)
    assert len(failed) >= 20  # the particle pools' allocations, then those of the pass
    for s in failed:
        for _ in range(2):
            assert_bins_equal(s.binParticles(), want)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_binning_after_a_failed_growth(cuda_lib, oracle, precision):
    """The failed pass is a later one, whose scene has spread over more pages."""
    rng = np.random.default_rng(4)
    few, many = SCENES["one-page"](rng), (20 + 30 * rng.random((900, 3))) * DX
    o = mpm.MpmSimulation(DX, precision=precision, lib=oracle)
    o.addParticles(many, None, 1.0, 1.0)
    want = o.binParticles()

    def prepare():
        s = mpm.MpmSimulation(DX, precision=precision, grid_log2=7)
        s.addParticles(few, None, 1.0, 1.0)
        s.binParticles()
        s.setParticles(X=many)
        return s

    failed = fail_each(cuda_lib, prepare)
    assert len(failed) >= 3  # neighbours, cells, pages
    for s in failed:
        for _ in range(2):
            assert_bins_equal(s.binParticles(), want)
