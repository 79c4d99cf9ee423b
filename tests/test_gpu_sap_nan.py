"""The collision-only step of the sweep-and-prune mode with positions that are not finite (a step
refuses them, the collision-only step does not look): the order is by interval minima (NaN before
or after the rest), an interval is walked until one starts past its maximum, which a NaN never
does, and a distance that is NaN is a hit."""
import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes

pytestmark = pytest.mark.gpu
F32 = np.float32


def swept(pos, radius, axis, nan_first):
    """Pairs in sweep order, in the arithmetic of the device (FP32, no contraction)."""
    lo = pos[:, axis] - radius
    order = np.argsort(lo, kind="stable")  # NaN last
    if nan_first:
        order = np.concatenate([order[np.isnan(lo[order])], order[~np.isnan(lo[order])]])
    pairs, checks = [], 0
    for x, a in enumerate(order):
        hi = pos[a, axis] + radius[a]
        for b in order[x + 1:]:
            if lo[b] > hi:
                break
            checks += 1
            d = pos[a] - pos[b]
            dist, r = F32(F32(d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]), F32(radius[a] + radius[b])
            if not dist > F32(r * r):
                pairs.append((a, b))
    return np.array(pairs, np.int32).reshape(-1, 2), checks


@pytest.mark.parametrize("n", [4, 40, 600])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_positions_that_are_not_finite(gpu, n, bad):
    b = scenes.SceneBuilder("line", scenes.baseline_params(broadphase=scenes.BROADPHASE_SAP))
    rs = np.random.default_rng(n)
    pos = np.stack([np.arange(n) * 0.9, rs.uniform(-0.1, 0.1, n), np.full(n, 2.0)], axis=1)
    b.bodies(np.full((n, 3), 0.8), np.ones(n), np.full(n, 0.5), pos)
    w = World(b.build())
    state = w.bodies()["pos"].copy()
    state[[1, n // 2, n - 1], 0] = bad
    state[1, 1] = bad
    w.write_bodies(pos=state)
    w.broadphase_only()
    radius = np.asarray(w.props["radius"], F32)
    with np.errstate(invalid="ignore", over="ignore"):
        wants = [swept(state, radius, 0, first) for first in (False, True)]  # a NaN mean: no axis beats x
    got, st = w.manifolds()["ab"], w.stats()
    assert any(np.array_equal(got, want) and (st["pair_checks"], st["sphere_hits"]) == (checks, len(want))
               for want, checks in wants)
    w.close()
