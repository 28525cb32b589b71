"""Particle fields between host arrays and the device: sizes from one particle
to many, every slot order, and Lame parameters set in place."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.scenes import jittered_box

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


# bytes of x (24 n) and C (72 n) around 2, 4 and 6 MB (whole pages and a few bytes off), and large
@pytest.mark.parametrize("n", [1, 29127, 29128, 58254, 58255, 87381, 87382, 174763, 400003])
def test_round_trip(cuda_lib, n):
    rng = np.random.default_rng(n)
    x = 0.3 + 0.4 * rng.random((n, 3))
    s = mpm.MpmSimulation(DX, precision="fp64", grid_log2=8)
    s.addParticles(x, None, 1.0, 1.0)
    a = {"X": x, "V": rng.standard_normal((n, 3)), "C": rng.standard_normal((n, 3, 3)), "F": rng.standard_normal((n, 3, 3))}
    s.binParticles()
    s.setParticles(**a)
    s.binParticles()  # the slots move
    for _ in range(2):
        b = s.getParticles()
        for k in a:
            np.testing.assert_array_equal(a[k], b[k])


def test_set_lame_in_place(cuda_lib):
    """Parameters of a range set before the first substep and on the device, in sorted slots, give the same substep;
    the phases of a split substep end, as with any edit."""
    x = jittered_box((6, 7, 5), DX, (0.3, 0.4, 0.3), 8, 2)
    V0, lo, hi = DX ** 3 / 8, 37, 900
    E = np.random.default_rng(1).uniform(5e3, 2e4, hi - lo)
    out = []
    for late in (False, True):
        s = mpm.MpmSimulation(DX, gravity=(0, -9.8, 0), precision="fp64", grid_log2=8)
        h = s.addParticles(x, np.random.default_rng(4).uniform(-1, 1, x.shape), 1000 * V0, V0)
        h.addFBasedMpmForce(mpm.NeoHookeanBorden(1e4, 0.3))
        if late:
            s.binParticles()
            s.particlesToGrid(1e-3)
        s.setYoungsModulus(E, 0.3, lo, hi)
        if late:
            with pytest.raises(abi.ZmpmError) as e:
                s.backwardEulerStep()
            assert e.value.status in (abi.NOT_READY, abi.BAD_ARG)
        for _ in range(2):
            assert s.advanceOneTimeStep(1e-3) == abi.OK
        out.append(s.getParticles())
    for k in out[0]:
        # the same FP64 sums in another order
        assert np.abs(out[0][k] - out[1][k]).max() <= 1e-11 * np.abs(out[0][k]).max(), k
