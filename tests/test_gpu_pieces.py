"""P2G, the Newton residual and the Hessian product where the split of the
particles over CTAs, warps and chunks can go wrong: single particles, cells
larger than a warp's chunk, one particle per cell, odd cuts of few groups over
many CTAs, and more groups than CTAs."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.scenes import jittered_box

pytestmark = pytest.mark.gpu

DX = 1.0 / 64
LO = (0.3, 0.4, 0.3)


def cell(n, seed=1):
    """n particles of one cell."""
    return (np.array([24.0, 28.0, 22.0]) + 0.5 + np.random.default_rng(seed).random((n, 3)) * 0.98) * DX


def spray(n, step, seed=2):
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return 0.2 + (step * g + 0.1 + 0.8 * np.random.default_rng(seed).random(g.shape)) * DX


SCENES = {
    "one": lambda: cell(1),
    "pair": lambda: cell(2),
    "cell-33": lambda: cell(33),
    "cell-600": lambda: cell(600),
    "sparse-cells": lambda: jittered_box((9, 5, 7), DX, LO, 1, 4),
    "dense-cells": lambda: jittered_box((4, 4, 4), DX, LO, 41, 5),
    "ragged": lambda: np.concatenate([jittered_box((11, 3, 6), DX, LO, 7, 6), cell(200, 7)]),
    "single-particle-groups": lambda: spray(9, 4),
    "more-groups-than-ctas": lambda: np.concatenate([spray(11, 4), spray(11, 4, 9), spray(11, 4, 10)]),
}


def make(lib, x, precision, layout, model):
    kw = {} if lib else {"grid_log2": 8, "layout": layout}
    s = mpm.MpmSimulation(DX, gravity=(0, -9.8, 0), precision=precision, lib=lib, **kw)
    V0 = DX ** 3 / 8
    rng = np.random.default_rng(3)
    h = s.addParticles(x, rng.uniform(-1, 1, x.shape), 1000 * V0, V0)
    h.addFBasedMpmForce(model(1e4, 0.3))
    s.addCollisionObject(mpm.AnalyticCollisionObject(mpm.HalfSpace((0, 0.42, 0), (0, 1, 0)), abi.SLIP))
    F = np.eye(3) + 0.1 * rng.standard_normal((len(x), 3, 3))
    s.setParticles(C=rng.uniform(-5, 5, (len(x), 3, 3)), F=F)
    return s


@pytest.mark.parametrize("scene", sorted(SCENES))
@pytest.mark.parametrize("precision,layout", [("fp64", "244"), ("fp64", "444"), ("mixed", "444"), ("mixed", "244")])
def test_transfers_and_products(cuda_lib, oracle, scene, precision, layout):
    x = SCENES[scene]().astype(np.float32).astype(np.float64)
    model = mpm.NeoHookeanBorden if scene in ("ragged", "cell-33") else mpm.FixedCorotated
    g, o = make(None, x, precision, layout, model), make(oracle, x, "fp64", layout, model)
    assert g.beginImplicit(1e-3) == o.beginImplicit(1e-3)
    # the two number their nodes by their own page shapes: compare by coordinate
    mg, vg, cg = g.getGrid()
    mo, vo, co = o.getGrid()
    ig, io = np.lexsort(cg.T), np.lexsort(co.T)
    np.testing.assert_array_equal(cg[ig], co[io])
    # FP32 terms of 6e-8 each, summed over at most a cell's particles; FP64 sums
    eps = 1e-13 if precision == "fp64" else 1e-6
    assert np.abs(mg[ig] - mo[io]).max() <= eps * mo.max()
    mom = np.abs(mo[io, None] * vo[io]).max()
    assert np.abs(mg[ig, None] * vg[ig] - mo[io, None] * vo[io]).max() <= 10 * eps * mom
    n = len(mg)
    dv = 0.1 * np.random.default_rng(8).standard_normal((n, 3))
    a, b = np.empty((n, 3)), np.empty((n, 3))
    a[ig], b[io] = dv, dv
    rg, ro = g.residual(a)[0], o.residual(b)[0]
    tol = 1e-10 if precision == "fp64" else 1e-5
    assert np.abs(rg[ig] - ro[io]).max() <= tol * np.abs(ro).max()
    pg, po = g.multiply(a, precision == "mixed"), o.multiply(b)
    assert np.abs(pg[ig] - po[io]).max() <= 2 * tol * np.abs(po).max()
