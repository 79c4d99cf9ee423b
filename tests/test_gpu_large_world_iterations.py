"""k_iterations, the iteration kernel of worlds beyond the wide kernel's body limit, on everything a
row can hold: small scenes beside a block of idle static bodies, which take a world past the limit
and change nothing else. Steps bit for bit against the CPU oracle, expired waits and taped steps."""
import dataclasses
import os
import re

import numpy as np
import pytest

from avbd_demo3d_b200 import World, _lib, scenes
from test_gpu_adjoint import _reference
from test_gpu_failure import MODES, recovers_bit_exact, step_status
from test_gpu_parity import assert_same_state, lockstep, static_pairs_scene
from test_gpu_wide_iterations import CASES, CSRC

pytestmark = pytest.mark.gpu


def constant(file, name):
    text = open(os.path.join(CSRC, file)).read()
    return eval(re.search(rf"\b{name} = ([^;,]+)[;,]", text).group(1).replace("(size_t)", ""))  # noqa: S307


LIMIT = constant("avbd_capi.cu", "WIDE_MAX_BODIES")


def beside_idle(scene, spare=30):
    """The scene and, far below it, a block of static boxes 1 m apart (0.5 m wide: no two meet)."""
    idle = LIMIT + spare - scene.n_bodies
    side = int(np.ceil(idle ** (1 / 3)))
    k = np.arange(idle)
    pos = np.stack([k % side, k // side % side, k // (side * side)], axis=1) - [side / 2, side / 2, side + 25.0]

    def grown(a, value):
        return np.concatenate([a, np.broadcast_to(np.asarray(value, a.dtype), (idle,) + a.shape[1:]).astype(a.dtype)])

    out = dataclasses.replace(
        scene, name=scene.name + "+idle", size=grown(scene.size, (0.5, 0.5, 0.5)), density=grown(scene.density, 0.0),
        friction=grown(scene.friction, 0.5), pos=np.concatenate([scene.pos, pos.astype(np.float32)]),
        vel=grown(scene.vel, 0.0), quat=grown(scene.quat, (0, 0, 0, 1)),
        shape=None if scene.shape is None else grown(scene.shape, 0),
        dims=None if scene.dims is None else grown(scene.dims, 0.0))
    assert out.n_bodies > LIMIT
    return out


SCENES = {k: v for k, v in CASES.items() if k != "more_chunks_than_warps"}
SCENES.update({
    "static_pairs": static_pairs_scene,
    "bridge": scenes.bridge,
    "springs": lambda: scenes.spring_chain(8),
    "spheres": lambda: scenes.sphere_pour(300),
    "mixed": lambda: scenes.mixed_drop(600, 6, 10, 0.05, extent=(14, 14, 12), seed=5),
    "pyramid": lambda: scenes.pyramid(12),
})


@pytest.mark.parametrize("name", sorted(SCENES))
def test_steps_match_oracle(gpu, name):
    lockstep(beside_idle(SCENES[name]()), 25)


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("scene", [lambda: scenes.stack_grid(8, 8, 8, seed=3), lambda: CASES["joints_37"]()])
def test_wait_expiry_fails_latches_and_recovers(gpu, mode, scene):
    sc = beside_idle(scene())
    w = World(sc)
    w.set_step_mode(MODES[mode])
    w.step(3)
    w.set_wait_limits(0, 1)
    assert step_status(w) == _lib.AVBD_ERR_STATE
    assert "iteration kernel wait expired" in w.last_error()
    assert w.lib.avbd_step(w.h, 1) == _lib.AVBD_ERR_LATCHED
    recovers_bit_exact(w, sc, steps=5)
    w.close()


def test_taped_steps_match_the_oracle_record(gpu):
    sc = beside_idle(scenes.tower(3, 3, 4, seed=4))
    w, plain = World(sc), World(sc)
    w.adjoint_forward(12, 5)
    plain.step(12)
    assert_same_state(w, plain, sc.name)
    ref = _reference(sc, 12)
    for s in range(12):
        t, r = w.adjoint_tape(s), ref.tape_step(s)
        assert t["nMan"] == r["nMan"]
        assert np.array_equal(t["body_flags"], r["body_flags"]) and np.array_equal(t["src"], r["src"])
        rf = r["flags"].astype(np.uint32)
        assert np.array_equal(t["flags"], (rf[..., 2] | (rf[..., 0] << 12) | (rf[..., 1] << 14)).astype(np.uint16))
    w.close()
    plain.close()
