"""The grid search's shared large-body part: bodies among many large ones, in their cells and on
the world's global list, fewer and more within reach than the lanes order together, against
the oracle (pairs, order, counters, states)."""
import numpy as np
import pytest

import checkers
from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu


def crowd(small, large, spread, speed, seed=3, box=False):
    """`small` little bodies amid `large` big ones (above the 95th percentile where they are few
    enough) in a cube of half-width `spread`; `speed` widens the large bodies' reach until
    they no longer fit cell lists and go to the global list."""
    rs = np.random.default_rng(seed)
    b = scenes.SceneBuilder("crowd", scenes.baseline_params(iterations=2))
    b.body((60, 60, 1), 0.0, 0.5, (0, 0, -0.5))
    kinds = np.array([0] * small + [1] * large)
    rs.shuffle(kinds)
    for k in kinds:
        pos = rs.uniform(-spread, spread, 3) + (0, 0, spread + 1)
        vel = rs.uniform(-speed, speed, 3)
        r = 0.1 if k == 0 else 0.8 + 0.3 * rs.random()
        if box:
            b.body((r, r, r), 1.0, 0.5, pos, vel)
        else:
            b.sphere(r, 1.0, 0.5, pos, vel)
    return b.build()


CASES = {
    "few_large": lambda: crowd(300, 10, 4.0, 1.0),
    "within_48": lambda: crowd(800, 40, 1.2, 1.0),
    "beyond_48": lambda: crowd(1600, 80, 1.0, 1.0),
    "global_list": lambda: crowd(800, 40, 3.0, 60.0),
    "global_beyond_48": lambda: crowd(1600, 80, 1.0, 80.0),
    "boxes": lambda: crowd(400, 20, 1.5, 20.0, box=True),
    "pour": lambda: scenes.sphere_pour(700, seed=9),
}


@pytest.mark.parametrize("mode", [scenes.BROADPHASE_GRID, scenes.BROADPHASE_LBVH])
@pytest.mark.parametrize("name", sorted(CASES))
def test_large_bodies(gpu, name, mode):
    sc = CASES[name]()
    so = CASES[name]()
    sc.params.broadphase = mode
    g, o = World(sc), checkers.World(so, "oracle", order_mode=1)
    for _ in range(2):
        g.broadphase_only()
        o.broadphase_only()
        mg, mo = g.manifolds(), o.manifolds()
        assert len(mg["ab"]) > 0 and np.array_equal(mg["ab"], mo["ab"]) and np.array_equal(mg["seq"], mo["seq"])
        st, c = g.stats(), o.counters()
        assert (st["sphere_hits"], st["constrained_hits"], st["manifold_count"]) == (c[1], c[2], c[4])
        if mode == scenes.BROADPHASE_GRID:
            assert st["pair_checks"] == c[0]
    for s in range(2):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, f"{name} step {s + 1}")
    g.close()
