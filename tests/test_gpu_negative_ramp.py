"""A penalty ramp below zero: contact penalties then change sign inside a step, which a world's
iterations have to keep whatever kernel they run in; bit for bit against the CPU oracle."""
import pytest

from avbd_demo3d_b200 import scenes
from test_gpu_parity import lockstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [-20.0, -1000.0])
def test_penalties_below_zero(gpu, beta):
    params = scenes.baseline_params()
    params.betaLin = beta
    lockstep(scenes.pyramid(6, params=params), 20)
