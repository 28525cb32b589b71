"""ADMM's global operator: the assembled node stencil that dense scenes take and
the matrix-free product that sparse ones keep, both against the oracle (which
assembles the reference's 125-entry rows)."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.scenes import jittered_box

pytestmark = pytest.mark.gpu

DX = 1.0 / 64
# launches per ADMM iteration: the stencil's product is part of the start kernel
STENCIL, MATRIX_FREE = 9, 10


def block(cells, ppc, seed):
    return jittered_box(cells, DX, (0.3, 0.4, 0.3), ppc, seed)


def spray(n, seed):
    """Single particles nine cells apart: every one touches eight pages of its own."""
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return 0.2 + (9 * g + np.random.default_rng(seed).random(g.shape)) * DX


def make(lib, x, precision, layout, iters):
    kw = {} if lib else {"grid_log2": 8, "layout": layout}
    s = mpm.MpmSimulation(DX, gravity=(0, -9.8, 0), precision=precision, lib=lib, **kw)
    V0 = DX ** 3 / 8
    v = np.random.default_rng(5).uniform(-0.5, 0.5, x.shape)
    h = s.addParticles(x, v, 1000 * V0, V0)
    h.addFBasedMpmForce(mpm.StvkWithHenckyIsotropic(2e4, 0.4))
    h.addFElasticNonequilibratedBasedMpmForce(mpm.StvkWithHencky(2e4, 0.4), 700.0, 700.0)
    s.addCollisionObject(mpm.AnalyticCollisionObject(mpm.HalfSpace((0, 0.42, 0), (0, 1, 0)), abi.SLIP))
    s.useAdmm(admm_max_iterations=iters, rho_scale=0.8, global_tolerance=1e-11)
    return s


def launches(x, precision, layout, iters):
    s = make(None, x, precision, layout, iters)
    assert s.advanceOneTimeStep(2e-3) == abi.OK
    return s.last_stats["kernel_launches"]


def expected(x, precision, layout):
    """The rule below 96 MB: the stencil where its bytes are at most 1 KB per particle, a group counting as 192."""
    page = np.array([2 if layout == "244" else 4, 4, 4])
    groups = np.unique(np.floor(x / DX - 0.5).astype(int) // page, axis=0)
    near = np.stack(np.meshgrid(*[np.arange(2)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pages = np.unique((groups[:, None] + near[None]).reshape(-1, 3), axis=0)
    size = len(pages) * 125 * page.prod() * (8 if precision == "fp64" else 4)
    return STENCIL if size <= 1024 * (len(x) + 192 * len(groups)) else MATRIX_FREE


# one cell (rows of one page corner), a page's edge, one past it, ragged and dense cells
@pytest.mark.parametrize("cells,ppc", [((1, 1, 1), 3), ((4, 4, 4), 8), ((5, 2, 9), 5), ((7, 6, 5), 27)])
@pytest.mark.parametrize("precision,layout", [("fp64", "244"), ("fp64", "444"), ("mixed", "444"), ("mixed", "244")])
def test_stencil_matches_oracle(cuda_lib, oracle, cells, ppc, precision, layout):
    x = block(cells, ppc, 3)
    assert launches(x, precision, layout, 2) - launches(x, precision, layout, 1) == expected(x, precision, layout)
    g, o = make(None, x, precision, layout, 6), make(oracle, x, "fp64", layout, 6)
    for _ in range(3):
        assert g.advanceOneTimeStep(2e-3) == o.advanceOneTimeStep(2e-3) == abi.OK
    a, b = g.getParticles(), o.getParticles()
    # mixed: FP32 coefficients (6e-8 relative each) through six solves, as the matrix-free product's FP32 terms
    tol = 1e-9 if precision == "fp64" else 1e-4
    for k in ("X", "V", "F"):
        assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sparse_scene_stays_matrix_free(cuda_lib, oracle, precision):
    x = spray(4, 2)
    assert launches(x, precision, "auto", 2) - launches(x, precision, "auto", 1) == MATRIX_FREE
    g, o = make(None, x, precision, "auto", 3), make(oracle, x, "fp64", "auto", 3)
    for _ in range(2):
        assert g.advanceOneTimeStep(2e-3) == o.advanceOneTimeStep(2e-3) == abi.OK
    a, b = g.getParticles(), o.getParticles()
    tol = 1e-9 if precision == "fp64" else 1e-4
    for k in ("X", "V", "F"):
        assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), k
