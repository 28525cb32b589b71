"""Binning by page and by radix sort give the same order: groups at the limits
that choose between them, and page tables left clean by every way out."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.test_gpu_binning import assert_bins_equal

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


def pair(oracle, x, precision, grid_log2=8, dx=DX):
    g = mpm.MpmSimulation(dx, precision=precision, grid_log2=grid_log2)
    o = mpm.MpmSimulation(dx, precision=precision, lib=oracle)
    for s in (g, o):
        s.addParticles(x, None, 1.0, 1.0)
    return g, o


# a group of 1, around a warp, and around the 2048 that one CTA orders; all of one cell or spread over a page
@pytest.mark.parametrize("n", [1, 31, 32, 33, 2047, 2048, 2049, 5000])
@pytest.mark.parametrize("spread", [0.9, 3.9])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_group_sizes(cuda_lib, oracle, n, spread, precision):
    rng = np.random.default_rng(n)
    x = (np.array([32.0, 32.0, 32.0]) + 0.55 + spread * rng.random((n, 3)) * [0.5, 1, 1]) * DX
    x = np.concatenate([x, (40 + 12 * rng.random((700, 3))) * DX]).astype(np.float32).astype(np.float64)
    g, o = pair(oracle, x[rng.permutation(len(x))], precision)
    b = o.binParticles()
    assert_bins_equal(g.binParticles(), b)
    assert_bins_equal(g.binParticles(), b)  # from sorted slots


# thousands of groups more than are ranked pairwise, one or two particles each
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_group_counts(cuda_lib, oracle, extra):
    g = np.stack(np.meshgrid(np.arange(32), np.arange(32), np.arange(17), indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(7)
    x = (4 * g[rng.permutation(len(g))[:16384 + extra]] + 8 + 0.6 + 2.8 * rng.random((16384 + extra, 3))) / 256
    x = np.concatenate([x, x[:500]]).astype(np.float32).astype(np.float64)
    a, o = pair(oracle, x, "mixed", 9, 1.0 / 256)
    assert_bins_equal(a.binParticles(), o.binParticles())


def test_tables_stay_clean(cuda_lib, oracle):
    """One context through both ways and an out-of-grid pass, in turn."""
    rng = np.random.default_rng(3)
    loose = (20 + 30 * rng.random((4000, 3))) * DX
    dense = (np.array([32.0, 32.0, 32.0]) + 0.55 + 0.9 * rng.random((4000, 3))) * DX
    bad = loose.copy()
    bad[17, 1] = -1.0
    g = mpm.MpmSimulation(DX, precision="fp64", grid_log2=8)
    g.addParticles(loose, None, 1.0, 1.0)
    for x in (loose, dense, bad, loose, bad, dense, loose):
        g.setParticles(X=x)
        if x is bad:
            with pytest.raises(abi.ZmpmError) as e:
                g.binParticles()
            assert e.value.status == abi.OUT_OF_GRID
            continue
        o = mpm.MpmSimulation(DX, precision="fp64", lib=oracle)
        o.addParticles(x, None, 1.0, 1.0)
        assert_bins_equal(g.binParticles(), o.binParticles())


# groups around the 8192 that are ranked pairwise, and a large group: a context takes the way of its last scene and
# finds back to the other
@pytest.mark.parametrize("groups", [8191, 8192, 8193])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_group_limit_and_way_back(cuda_lib, oracle, groups, precision):
    page = np.array([2, 4, 4] if precision == "fp64" else [4, 4, 4])
    g = np.stack(np.meshgrid(np.arange(20), np.arange(20), np.arange(21), indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(11)
    many = page * g[rng.permutation(len(g))[:groups]] + 8 + 0.6 + (page - 1.2) * rng.random((groups, 3))
    few = 40 + 8 * rng.random((groups, 3))
    few[2200:] += 30 * rng.random((groups - 2200, 3))
    cell = 40.55 + 0.9 * rng.random((groups, 3))  # one group of all
    s = mpm.MpmSimulation(1.0 / 256, precision=precision, grid_log2=8)
    s.addParticles(many / 256, None, 1.0, 1.0)
    for x in (many, few, cell, many, cell, few, few, many):
        x = (x / 256).astype(np.float32).astype(np.float64)
        s.setParticles(X=x)
        o = mpm.MpmSimulation(1.0 / 256, precision=precision, lib=oracle)
        o.addParticles(x, None, 1.0, 1.0)
        for _ in range(2):
            assert_bins_equal(s.binParticles(), o.binParticles())


def test_large_scenes_count_their_pages_once(cuda_lib):
    """A scene for the radix way is not put through the page counts again on every pass."""
    rng = np.random.default_rng(5)
    s = mpm.MpmSimulation(DX, precision="fp64", grid_log2=7)
    s.addParticles((32.55 + 0.9 * rng.random((4000, 3))) * DX, None, 1.0, 1.0)
    s.useExplicit()
    n = []
    for _ in range(3):
        assert s.advanceOneTimeStep(1e-4) == abi.OK
        n.append(s.last_stats["kernel_launches"])
    assert n[1] == n[2] == n[0] - 3  # the counts, the pages, the unmarking


@pytest.mark.parametrize("precision,nodes_per_page", [("fp64", 32), ("mixed", 64)])
def test_two_page_tables(cuda_lib, precision, nodes_per_page):
    """A context holds two words per page of the grid, not more (the tables are 8.6 GB each at grid_log2 = 12, FP64)."""
    import torch
    table = 4 * (1 << 30) // nodes_per_page
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s = mpm.MpmSimulation(DX, precision=precision, grid_log2=10)
    assert free - torch.cuda.mem_get_info()[0] < 2.8 * table + (8 << 20)  # with the rounding up of allocations
    s.close()
