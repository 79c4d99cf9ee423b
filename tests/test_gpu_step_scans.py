"""A device step's one-block scans and fused launches around the sizes where they turn (tiles of
4,096 values, the 32,768 beyond which the library scan takes over), against the synchronous
step, which scans and launches separately."""
import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,height,steps", [
    (1, 1, 1, 4), (1, 2, 1, 4), (2, 1, 5, 4),
    (16, 16, 16, 4),    # one tile of grid entries, about
    (16, 20, 16, 3),    # 32,768 force-list entries (with the spare manifolds), about: below
    (18, 18, 16, 3),    # and above
    (25, 26, 16, 3),    # 32,768 manifolds with the spare ones, about: below
    (26, 27, 16, 3),    # and above
    (64, 32, 16, 2),    # 32,768 grid entries, about: below
    (64, 35, 16, 2),    # and above
])
@pytest.mark.parametrize("mode", [scenes.BROADPHASE_GRID, scenes.BROADPHASE_LBVH])
def test_device_step_is_host_step(gpu, nx, ny, height, steps, mode):
    if mode == scenes.BROADPHASE_LBVH and nx > 26:
        pytest.skip("the grid form covers the size")
    scene = scenes.stack_grid(nx, ny, height, seed=nx + ny, params=scenes.baseline_params(broadphase=mode))
    a, b = World(scene), World(scene)
    b.set_step_mode(World.STEP_HOST)
    a.step(steps, sync=False)
    b.step(steps)
    assert_same_state(a, b, scene.name)
    sa, sb = a.stats(), b.stats()
    assert sa["device_steps"] == steps and sa["redone_steps"] == 0
    for k in ("pair_checks", "sphere_hits", "constrained_hits", "manifolds_created", "manifold_count", "colours"):
        assert sa[k] == sb[k], k
    a.close()
    b.close()


def test_counts_survive_between_device_and_host_steps(gpu):
    """The device's counts are written anew only when the host's differ: alternating the step
    forms, reloading and editing leaves them in step."""
    scene = scenes.mixed_drop(400, 4, 8, 0.05, extent=(12, 12, 10), seed=2)
    a, b = World(scene), World(scene)
    b.set_step_mode(World.STEP_HOST)
    for k in range(12):
        a.set_step_mode(World.STEP_HOST if k % 3 == 1 else World.STEP_DEVICE)
        a.step(1 + k % 2, sync=False)
        b.step(1 + k % 2)
        if k == 5:
            for w in (a, b):
                w.add_joint(0, 1, (0, 0, 1), (0, 0, -1))
        if k == 8:
            for w in (a, b):
                w.broadphase_only()
        if k == 9:
            a.reload()
            b.reload()
        assert_same_state(a, b, f"round {k}")
        assert a.next_seq() == b.next_seq()
    a.close()
    b.close()
