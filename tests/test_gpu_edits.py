"""Edits of a scene that is on the device."""
import numpy as np
import pytest

from ziran2019_b200 import abi, mpm
from tests.scenes import jittered_box

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


def make():
    x = jittered_box((5, 6, 4), DX, (0.3, 0.4, 0.3), 8, 2)
    V0 = DX ** 3 / 8
    s = mpm.MpmSimulation(DX, gravity=(0, -9.8, 0), precision="fp64", grid_log2=7)
    h = s.addParticles(x, np.random.default_rng(4).uniform(-1, 1, x.shape), 1000 * V0, V0)
    h.addFBasedMpmForce(mpm.NeoHookeanBorden(1e4, 0.3))
    return s


@pytest.mark.parametrize("hi", [0, 1, None])
def test_checkpoint_does_not_load_over_new_moduli(cuda_lib, hi):
    """save, setYoungsModulus, load: the load would put the old moduli back unseen, so it is refused, and the new ones
    stand.  After a substep it loads, old moduli and all."""
    s = make()
    s.checkpointSave(0)
    before = s.getParticles()
    s.setYoungsModulus(4e4, 0.3, 0, hi)
    with pytest.raises(abi.ZmpmError) as e:
        s.checkpointLoad(0)
    assert e.value.status == abi.BAD_ARG
    for k, a in s.getParticles().items():
        np.testing.assert_array_equal(a, before[k])
    assert s.advanceOneTimeStep(1e-3) == abi.OK
    stiff = s.getParticles()
    s.checkpointLoad(0)
    assert s.advanceOneTimeStep(1e-3) == abi.OK
    soft = s.getParticles()
    assert (hi == 0) == (np.abs(stiff["F"] - soft["F"]).max() <= 1e-11)
    # saving counts as a run: the checkpoint holds the new moduli
    s.setYoungsModulus(4e4, 0.3, 0, hi)
    s.checkpointSave(0)
    s.checkpointLoad(0)
