"""The sweep-and-prune sweep where its parts and searches turn: candidate stretches around
multiples of the part length, minima equal to a maximum at zero, many worlds; pairs, order and
counters against the CPU oracle, in both step forms."""
import numpy as np
import pytest

import checkers
from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state, lockstep

pytestmark = pytest.mark.gpu


def sap(**kw):
    return scenes.baseline_params(broadphase=scenes.BROADPHASE_SAP, **kw)


def row(n, pitch=0.9):
    """n boxes in a line on a ground under all of them: its interval holds every other body."""
    b = scenes.SceneBuilder(f"row{n}", sap())
    b.body((2 * n * pitch + 10, 20, 1), 0.0, 0.5, (0, 0, -0.5))
    b.bodies(np.full((n, 3), 0.8), np.ones(n), np.full(n, 0.5),
             np.stack([(np.arange(n) - n / 2) * pitch, np.zeros(n), np.full(n, 0.4)], axis=1))
    return b.build()


def touching_at_zero():
    """Intervals that end and begin at zero, of either sign (spheres of radius 1 at -1 and 1)."""
    b = scenes.SceneBuilder("zero", sap())
    b.body((40, 4, 1), 0.0, 0.5, (0, 0, -0.5))
    for x in (-1.0, 1.0, -3.0, 3.0):
        b.sphere(1.0, 1.0, 0.5, (x, 0.0, 1.0))
    return b.build()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 1057, 2100])
def test_sweep_parts(gpu, n):
    sc = row(n)
    g, o = World(sc), checkers.World(sc, "oracle", order_mode=1)
    for _ in range(2):
        g.broadphase_only()
        o.broadphase_only()
        mg, mo = g.manifolds(), o.manifolds()
        assert np.array_equal(mg["ab"], mo["ab"]) and np.array_equal(mg["seq"], mo["seq"])
        st, c = g.stats(), o.counters()
        assert (st["pair_checks"], st["sphere_hits"], st["constrained_hits"], st["manifold_count"]) == \
            (c[0], c[1], c[2], c[4])
    for s in range(3):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, f"{sc.name} step {s + 1}")
    g.close()


def test_touching_at_zero(gpu):
    sc = touching_at_zero()
    g, o = World(sc), checkers.World(sc, "oracle", order_mode=1)
    g.broadphase_only()
    o.broadphase_only()
    assert np.array_equal(g.manifolds()["ab"], o.manifolds()["ab"])
    assert g.stats()["pair_checks"] == o.counters()[0]
    g.close()
    lockstep(sc, 10)


def test_device_steps_are_host_steps(gpu):
    """Steps that keep their counts on the device, queued without waiting, against the
    synchronous form: joints that break and pairs beyond the manifold room are redone."""
    worlds = [scenes.stack_grid(3, 3, 5, seed=1, params=sap()), scenes.breakable(params=scenes.Params(broadphase=scenes.BROADPHASE_SAP)),
              scenes.mixed_drop(400, 4, 8, 0.05, extent=(12, 12, 10), seed=2, params=sap()),
              scenes.round_mix(60, seed=4, cols=3, params=sap())]
    for scene, spare in [(worlds, 0), (scenes.stack_grid(6, 6, 8, seed=3, params=sap()), 1), (worlds[1], 0)]:
        a, b = World(scene), World(scene)
        a.set_manifold_headroom(spare)
        b.set_step_mode(World.STEP_HOST)
        for s in range(6):
            a.step(10, sync=False)
            b.step(10)
            assert_same_state(a, b, f"step {10 * s + 10}")
        assert a.stats()["device_steps"] == 60
        a.close()
        b.close()
