"""When ADMM's global operator stays matrix-free: large sparse scenes, whose
coefficients no longer fit the L2 cache, and a device without room for them."""
import numpy as np
import pytest

from ziran2019_b200 import abi
from tests.test_gpu_stencil import MATRIX_FREE, STENCIL, block, launches, make
from tests.test_gpu_stencil import DX

pytestmark = pytest.mark.gpu


def grid(n, step, seed):
    """Single particles `step` cells apart."""
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    return 0.3 + (step * g + np.random.default_rng(seed).random(g.shape)) * DX


# (MB of coefficients, bytes per unit): 30, 560 | 182, 490 | 164, 370 | 200, 290
@pytest.mark.parametrize("precision,n,step,ways", [("fp64", (8, 5, 8), 4, STENCIL), ("fp64", (16, 9, 16), 4, MATRIX_FREE),
                                                   ("mixed", (16, 9, 16), 5, MATRIX_FREE), ("mixed", (20, 12, 20), 4, STENCIL)])
def test_large_sparse_scenes(cuda_lib, oracle, precision, n, step, ways):
    x = grid(n, step, 3)
    assert launches(x, precision, "auto", 2) - launches(x, precision, "auto", 1) == ways
    g, o = make(None, x, precision, "auto", 2), make(oracle, x, "fp64", "auto", 2)
    for _ in range(2):
        assert g.advanceOneTimeStep(2e-3) == o.advanceOneTimeStep(2e-3) == abi.OK
    a, b = g.getParticles(), o.getParticles()
    tol = 1e-9 if precision == "fp64" else 1e-4  # as in test_gpu_stencil
    for k in ("X", "V", "F"):
        assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_room_for_the_coefficients(cuda_lib, oracle, precision):
    """Each allocation of a first ADMM substep failing in turn: without the operator's two arrays the substep runs
    matrix-free, without any other it reports the error; the context goes on as if nothing had been."""
    x, iters = block((7, 6, 5), 27, 3), 3  # two iterations launch as many kernels either way
    want = make(None, x, precision, "auto", iters)
    assert want.advanceOneTimeStep(2e-3) == abi.OK
    full = want.last_stats["kernel_launches"]
    o = make(oracle, x, "fp64", "auto", iters)
    for _ in range(2):
        assert o.advanceOneTimeStep(2e-3) == abi.OK
    b = o.getParticles()
    tol = 1e-9 if precision == "fp64" else 1e-4
    free, n = 0, 0
    while True:
        s = make(None, x, precision, "auto", iters)
        cuda_lib.fail_allocation(n + 1)
        try:
            rc = s.advanceOneTimeStep(2e-3)
        except abi.ZmpmError as e:
            rc = e.status
        untouched = cuda_lib.fail_allocation(0) == abi.OK and rc == abi.OK and s.last_stats["kernel_launches"] == full
        if untouched:
            break  # fewer allocations than n + 1
        n += 1
        if rc == abi.OK:
            free += 1
        else:
            assert rc == abi.CUDA_ERROR
            assert s.advanceOneTimeStep(2e-3) == abi.OK
        assert s.advanceOneTimeStep(2e-3) == abi.OK
        a = s.getParticles()
        for k in ("X", "V", "F"):
            assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), (n, k)
    assert free == 2 and n > 30


@pytest.mark.parametrize("cells,ppc", [((9, 7, 11), 8), ((12, 12, 12), 1)])
def test_mixed_substep_repeats(cuda_lib, cells, ppc):
    """MIXED sums the FP32 coefficients in the order its atomics arrive: from one checkpoint the velocities repeat to
    FP32's rounding and the Krylov counts to one iteration."""
    s = make(None, block(cells, ppc, 4), "mixed", "auto", 6)
    s.checkpointSave(0)
    assert s.advanceOneTimeStep(2e-3) == abi.OK
    s.checkpointSave(0)
    v, counts = [], []
    for _ in range(6):
        s.checkpointLoad(0)
        assert s.advanceOneTimeStep(2e-3) == abi.OK
        v.append(s.getParticles()["V"])
        counts.append(s.last_stats["krylov_iterations"])
    assert max(counts) - min(counts) <= 1
    assert max(np.linalg.norm(a - v[0]) for a in v) <= 2 * 2.0 ** -24 * np.linalg.norm(v[0])
