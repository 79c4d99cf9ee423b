"""The sweep-and-prune sweep where its split turns: intervals at the most candidates a warp takes
alone, at the block's tiles, several long ones in one block, worlds at the sizes where an interval
gets more or fewer warps, and batches that mix worlds of a few bodies with a large one; pairs,
order and counters against the CPU oracle."""
import numpy as np
import pytest

import checkers
from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state
from test_gpu_sap_sweep import row, sap

pytestmark = pytest.mark.gpu


def wall(n):
    """n boxes in the plane across the sweep axis: every interval holds all the later ones."""
    b = scenes.SceneBuilder(f"wall{n}", sap())
    b.body((400, 4, 1), 0.0, 0.5, (0, 0, -0.5))
    b.body((1, 1, 1), 1.0, 0.5, (-150, 0, 0.5))  # two far ones make x the sweep axis
    b.body((1, 1, 1), 1.0, 0.5, (150, 0, 0.5))
    k = np.arange(n)
    b.bodies(np.full((n, 3), 0.8), np.ones(n), np.full(n, 0.5),
             np.stack([0.001 * (k % 7), (k % 6 - 2.5) * 0.9, 0.4 + 0.79 * (k // 6)], axis=1))
    return b.build()


def same_pairs(sc, oracles):
    g = World(sc)
    for _ in range(2):
        g.broadphase_only()
        want_ab, want_c, first = [], np.zeros(3, np.int64), 0
        for o in oracles:
            o.broadphase_only()
            want_ab.append(o.manifolds()["ab"] + first)
            want_c += np.asarray(o.counters()[:3], np.int64)
            first += o.n
        mg, st = g.manifolds(), g.stats()
        assert np.array_equal(mg["ab"], np.concatenate(want_ab))
        assert (st["pair_checks"], st["sphere_hits"], st["constrained_hits"]) == tuple(want_c)
    return g


@pytest.mark.parametrize("n", [510, 511, 512, 513, 1534, 1535, 1536, 1537, 2560])
def test_one_long_interval(gpu, n):
    sc = row(n)
    o = checkers.World(sc, "oracle", order_mode=1)
    g = same_pairs(sc, [o])
    for s in range(2):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, f"{sc.name} step {s + 1}")
    g.close()


@pytest.mark.parametrize("n", [514, 600, 1100])
def test_many_long_intervals_in_a_block(gpu, n):
    sc = wall(n)
    o = checkers.World(sc, "oracle", order_mode=1)
    g = same_pairs(sc, [o])
    for s in range(2):
        g.step(1)
        o.step(1)
        assert_same_state(g, o, f"{sc.name} step {s + 1}")
    g.close()


@pytest.mark.parametrize("bodies", [148, 149, 296, 297, 592, 593, 1184, 1185, 2368, 2369, 4737])
def test_warps_to_an_interval(gpu, bodies):
    for sc in (row(bodies - 1), scenes.stack_grid(1, (bodies - 1) // 8, 8, seed=2, params=sap())):
        o = checkers.World(sc, "oracle", order_mode=1)
        g = same_pairs(sc, [o])
        for s in range(2):
            g.step(1)
            o.step(1)
            assert_same_state(g, o, f"{sc.name} step {s + 1}")
        g.close()


def test_small_worlds_beside_a_large_one(gpu):
    small = [scenes.pyramid(k, params=sap()) for k in (1, 2, 3, 4)]
    worlds = small * 5 + [wall(700)] + small + [row(40), scenes.stack_grid(5, 5, 6, seed=2, params=sap())] + small * 9
    same_pairs(worlds, [checkers.World(sc, "oracle", order_mode=1) for sc in worlds]).close()
