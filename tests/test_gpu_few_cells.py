"""Groups of few cells, where a CTA's warps share the particles instead of the
cells: one to nine cells (the rule changes at eight), groups cut by several
CTAs, and warps left without a particle."""
import numpy as np
import pytest

from tests import test_gpu_pieces as pieces

pytestmark = pytest.mark.gpu


def cells(ncell, n, seed):
    """n particles spread unevenly over ncell cells of one page."""
    rng = np.random.default_rng(seed)
    w = rng.random(ncell) ** 3 + 0.01
    c = np.concatenate([np.arange(min(n, ncell)), rng.choice(ncell, max(0, n - ncell), p=w / w.sum())])
    off = np.stack([c & 1, (c >> 1) & 3, c >> 3], -1)
    return (np.array([24.0, 28.0, 20.0]) + 0.51 + off + rng.random((n, 3)) * 0.98) * pieces.DX


@pytest.mark.parametrize("ncell", [2, 3, 7, 8, 9])
@pytest.mark.parametrize("n", [3, 130, 701, 3000])
@pytest.mark.parametrize("precision,layout", [("fp64", "244"), ("fp64", "444"), ("mixed", "444"), ("mixed", "244")])
def test_few_cells(cuda_lib, oracle, monkeypatch, ncell, n, precision, layout):
    monkeypatch.setitem(pieces.SCENES, "few-cells", lambda: cells(ncell, n, 10 * ncell + n))
    pieces.test_transfers_and_products(cuda_lib, oracle, "few-cells", precision, layout)
