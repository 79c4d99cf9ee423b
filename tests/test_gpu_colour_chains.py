"""The greedy colouring's chain shortcut: chains that start, branch, double and cross warps at
awkward places, against the oracle's sequential greedy colouring (colours, rounds and states)."""
import pytest

import checkers
from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu


def chain(n, extra=(), doubled=False, reverse=False, static=()):
    """n links in a row above a ground, each jointed to the one before; `extra`: further joints
    (i, j); `doubled`: two joints per link; `reverse`: created from the far end, so every link's
    neighbour is newer; `static`: links without mass."""
    b = scenes.SceneBuilder(f"chain{n}", scenes.baseline_params(iterations=3))
    b.body((4 * n + 20, 40, 1), 0.0, 0.5, (0, 0, -0.5))
    at = {}
    for k in (reversed(range(n)) if reverse else range(n)):
        at[k] = b.body((0.8, 0.4, 0.4), 0.0 if k in static else 1.0, 0.5, (k - n / 2, 0, 3.0))
    for k in range(1, n):
        for y in ((-0.15, 0.15) if doubled else (0.0,)):
            b.joint(at[k - 1], at[k], (0.5, y, 0), (-0.5, y, 0))
    for i, j in extra:
        b.spring(at[i], at[j], (0, 0, 0.2), (0, 0, 0.2), 50.0)
    return b.build()


CASES = {
    "pair": lambda: chain(2),
    "one_warp": lambda: chain(31),
    "warp_edges": lambda: chain(33),
    "many_warps": lambda: chain(700),
    "doubled_joints": lambda: chain(100, doubled=True),
    "newer_neighbours": lambda: chain(150, reverse=True),
    "breaks": lambda: chain(130, static=(0, 31, 32, 64, 100)),
    "ring": lambda: chain(97, extra=((0, 96),)),
    "branches": lambda: chain(200, extra=tuple((k, k + 7) for k in range(3, 190, 11))),
    "long_branches": lambda: chain(300, extra=tuple((k, k + 70) for k in range(0, 220, 31))),
    "star": lambda: chain(64, extra=tuple((20, k) for k in range(24, 60))),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_chain_colours(gpu, name):
    sc = CASES[name]()
    g, o = World(sc), checkers.World(sc, "oracle", order_mode=1)
    for s in range(2):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, f"{name} step {s + 1}")
    g.close()
