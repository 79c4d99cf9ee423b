"""The grid search's counting and emitting passes where their blocks go round more than once, in a
batch large enough to launch more blocks than the usual most, and where lanes find more pairs
than they record and search again while emitting."""
import numpy as np
import pytest

import checkers
from avbd_demo3d_b200 import World, scenes

pytestmark = pytest.mark.gpu


def clump(count, cells, seed=2):
    """`cells` clumps of `count` overlapping boxes, a cell wide: a lane meets its whole clump."""
    rs = np.random.default_rng(seed)
    b = scenes.SceneBuilder(f"clump{count}", scenes.baseline_params())
    b.body((80, 80, 1), 0.0, 0.5, (0, 0, -0.5))
    centre = np.stack([np.arange(cells) * 6.0 - 3.0 * cells, np.zeros(cells), np.full(cells, 2.0)], axis=1)
    pos = np.repeat(centre, count, axis=0) + rs.uniform(-0.3, 0.3, (count * cells, 3))
    b.bodies(np.full((len(pos), 3), 0.8), np.ones(len(pos)), np.full(len(pos), 0.5), pos)
    return b.build()


@pytest.mark.parametrize("count,cells", [(8, 3), (9, 3), (10, 3), (40, 4), (200, 1)])
def test_more_pairs_than_a_lane_records(gpu, count, cells):
    sc = clump(count, cells)
    g, o = World(sc), checkers.World(sc, "oracle", order_mode=1)
    for _ in range(2):
        g.broadphase_only()
        o.broadphase_only()
        mg, mo = g.manifolds(), o.manifolds()
        assert len(mg["ab"]) > 0 and np.array_equal(mg["ab"], mo["ab"]) and np.array_equal(mg["seq"], mo["seq"])
        st, c = g.stats(), o.counters()
        assert (st["pair_checks"], st["sphere_hits"], st["constrained_hits"]) == tuple(c[:3])
    g.close()


@pytest.mark.parametrize("worlds", [25, 235, 480])  # 1, 7 and 15 rounds of the usual most blocks
def test_batch_is_its_worlds(gpu, worlds):
    one = scenes.stack_grid(10, 5, 12, seed=5)
    a, b = World(one), World([one] * worlds)
    for w in (a, b):
        w.broadphase_only()
    sa, sb = a.stats(), b.stats()
    for k in ("pair_checks", "sphere_hits", "constrained_hits", "manifold_count"):
        assert sb[k] == worlds * sa[k], k
    want, got = a.manifolds()["ab"], b.manifolds()["ab"]
    per = len(want)
    # a batch lists the grid entries' pairs of every world before the pairs of large bodies
    order = np.argsort(got[:, 0] // one.n_bodies, kind="stable")
    shifted = want[None] + (np.arange(worlds) * one.n_bodies)[:, None, None]
    assert np.array_equal(got[order].reshape(worlds, per, 2), shifted)
    a.close()
    b.close()
