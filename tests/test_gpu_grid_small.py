"""The one-block grid of a small world around the sizes where it turns: one entry a thread up to
1,024 binned bodies, four up to 4,096, the launches beyond, against the synchronous step, which
always grids with launches."""
import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state


def binned_count(scene):
    """Bodies at or below the 95th-percentile bounding radius."""
    half = np.asarray(scene.size, np.float32) * np.float32(0.5)
    r = np.sqrt((half * half).sum(axis=1))
    return int((r <= np.sort(r)[min(len(r) - 1, len(r) * 95 // 100)]).sum())


def drop(n, extent):
    return scenes.mixed_drop(n, 0, 1, 0.0, extent=extent, seed=n)


SIZES = [(1075, (22, 22, 10), 1023), (1076, (22, 22, 10), 1024), (1077, (22, 22, 10), 1025),
         (4309, (40, 40, 14), 4095), (4310, (40, 40, 14), 4096), (4311, (40, 40, 14), 4097)]


@pytest.mark.parametrize("n,extent,binned", SIZES)
def test_sizes_straddle_the_limits(n, extent, binned):
    assert binned_count(drop(n, extent)) == binned


@pytest.mark.gpu
@pytest.mark.parametrize("n,extent,binned", SIZES)
def test_one_block_grid_is_launched_grid(gpu, n, extent, binned):
    scene = drop(n, extent)
    a, b = World(scene), World(scene)
    b.set_step_mode(World.STEP_HOST)
    for k in range(4):
        a.step(10, sync=False)
        b.step(10)
        assert_same_state(a, b, f"{n} bodies, round {k}")
        sa, sb = a.stats(), b.stats()
        for key in ("pair_checks", "sphere_hits", "manifold_count", "colours"):
            assert sa[key] == sb[key], key
    assert sa["manifold_count"] > 0
    a.close()
    b.close()
