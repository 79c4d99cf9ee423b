"""Worlds of one layer, where the iteration kernel is chosen by the colours of the step before: at
the most bodies the wide kernel's warps take in one round, and in worlds whose colours come and
go, bit for bit against the per-colour launches (which share none of either kernel's data flow)."""
import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes
from test_gpu_adjoint import _gpu_gradient, _reference, _target
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu


def layer(n, falling=0, height=2.0):
    """n boxes side by side on the ground, `falling` of them with a box above it."""
    b = scenes.SceneBuilder(f"layer{n}", scenes.baseline_params())
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    pos = np.stack([(k % side - side / 2) * 1.5, (k // side - side / 2) * 1.5, np.full(n, 0.5)], axis=1)
    above = pos[np.linspace(0, n - 1, falling).astype(int)] + [0.1, 0.0, height]
    b.body((2 * side + 10, 2 * side + 10, 1), 0.0, 0.5, (0, 0, -0.5))
    every = np.concatenate([pos, above])
    b.bodies(np.ones((len(every), 3)), np.ones(len(every)), np.full(len(every), 0.5), every)
    return b.build()


@pytest.mark.parametrize("n", [7103, 7104, 7105, 8200])
@pytest.mark.parametrize("mode", [World.STEP_DEVICE, World.STEP_HOST])
def test_one_layer(gpu, n, mode):
    scene = layer(n)
    a, b = World(scene), World(scene)
    a.set_step_mode(mode)
    b.set_iteration_mode(0)
    for k in (1, 2, 5):
        a.step(k, sync=False)
        b.step(k)
        assert_same_state(a, b, f"{scene.name} {k} steps")
    assert a.colours()[1] == 1
    a.close()
    b.close()


@pytest.mark.parametrize("mode", [World.STEP_DEVICE, World.STEP_HOST])
def test_colours_that_come_and_go(gpu, mode):
    """Boxes fall on the layer (a second colour), are lifted off it again, and the world is
    loaded anew: the choice follows late, the bits do not depend on it."""
    scene = layer(7300, falling=40)
    a, b = World(scene), World(scene)
    a.set_step_mode(mode)
    b.set_iteration_mode(0)
    colours = set()
    for round_ in range(2):
        for k in (4, 20, 3, 3):
            a.step(k, sync=False)
            b.step(k)
            assert_same_state(a, b, f"round {round_}, {k} steps")
            colours.add(a.colours()[1])
        pos = b.bodies()["pos"].copy()
        pos[1:41, 2] += 5.0 if pos[1, 2] > 1.2 else 0.0
        pos[-40:, 2] += 5.0 if pos[-1, 2] > 1.2 else 0.0
        for w in (a, b):
            w.write_bodies(pos=pos)
        for k in (1, 2):
            a.step(k, sync=False)
            b.step(k)
            assert_same_state(a, b, f"round {round_}, lifted, {k} steps")
            colours.add(a.colours()[1])
        a.reload()
        b.reload()
    assert colours >= {1, 2}
    a.close()
    b.close()


def test_differentiable_steps_of_one_layer(gpu):
    """Taped steps on both sides of the choice (the first, of no known colours, in the wide kernel):
    the plain step's bits, the branches the oracle takes, and the oracle's gradient within the
    tolerance of the other gradient tests (the same map in 64 bits, sums in another order)."""
    scene = layer(7300)
    steps, target = 5, _target(scene)
    w, loss, g, _, _, _, _, _, _ = _gpu_gradient(scene, steps, 2, target)
    plain, ref = World(scene), _reference(scene, steps)
    plain.step(steps)
    assert_same_state(w, plain, scene.name)
    for s in range(steps):
        t, r = w.adjoint_tape(s), ref.tape_step(s)
        assert t["nMan"] == r["nMan"]
        assert np.array_equal(t["body_flags"], r["body_flags"]) and np.array_equal(t["src"], r["src"])
        rf = r["flags"].astype(np.uint32)
        assert np.array_equal(t["flags"], (rf[..., 2] | (rf[..., 0] << 12) | (rf[..., 1] << 14)).astype(np.uint16))
    rloss, rg = ref.adj_gradient(ref.adj_theta0(), target)
    assert loss == pytest.approx(rloss, rel=1e-10)
    assert np.linalg.norm(g - rg) <= 1e-6 * np.linalg.norm(rg)
    w.close()
    plain.close()
