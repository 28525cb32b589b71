"""MIXED P2G rounds no more than w_ip m_p (v_p + C_p (x_i - x_p)) formed and
rounded term by term in FP32: the affine form it uses is taken about the
stencil's centre (about a corner node its terms are twice as large)."""
import numpy as np
import pytest

from ziran2019_b200 import mpm

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


def scene(seed):
    """Cells of 8 particles; fractions, velocities and gradients that FP32 holds exactly."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in (9, 7, 8)], indexing="ij"), -1).reshape(-1, 3)
    base = 20 + np.repeat(g, 8, 0)
    P = len(base)
    return base, 0.5 + rng.integers(1, 4096, (P, 3)) / 4096, rng.integers(-64, 64, (P, 3)) / 64, rng.integers(-8192, 8192, (P, 3, 3)) / 64


def momentum(base, fr, v, C, t):
    """Grid momentum for unit masses; the terms in precision t, their sums in FP64."""
    fr, v, C = fr.astype(t), v.astype(t), C.astype(t)
    z, d1 = t(1.5) - fr, fr - t(1)
    zz = t(0.5) + d1
    w = np.stack([t(0.5) * z * z, t(0.75) - d1 * d1, t(0.5) * zz * zz], 1)
    out = np.zeros((*(base.max(0) + 4), 3))
    for o in np.ndindex(3, 3, 3):
        xi = (np.array(o, dtype=t) - fr) * t(DX)
        term = (w[:, o[0], 0] * w[:, o[1], 1] * w[:, o[2], 2])[:, None] * (v + (C * xi[:, None, :]).sum(2, dtype=t))
        np.add.at(out, tuple((base + o).T), term.astype(np.float64))
    return out


@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("layout", ["244", "444"])
def test_mixed_p2g_rounds_like_its_terms(cuda_lib, seed, layout):
    base, fr, v, C = scene(seed)
    s = mpm.MpmSimulation(DX, gravity=(0, 0, 0), precision="mixed", grid_log2=7, layout=layout)
    s.addParticles((base + fr) * DX, v, 1.0, 1.0)
    s.setParticles(C=C)
    s.beginImplicit(1e-4)
    m, vg, c = s.getGrid()
    got = np.zeros((*(base.max(0) + 4), 3))
    got[tuple(c.T)] = m[:, None] * vg
    want, terms = momentum(base, fr, v, C, np.float64), momentum(base, fr, v, C, np.float32)
    # a node sums a cell's terms in FP32 (8 of them: about half an ulp more each way), all else in FP64
    assert np.linalg.norm(got - want) <= 1.5 * np.linalg.norm(terms - want)
