"""Where the backward takes its last segment's snapshots from: the forward, its own replay (a
segment beyond what a forward keeps), and again after another backward has used the buffers."""
import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes
from test_gpu_adjoint import _gpu_gradient, _reference, _target
from test_gpu_large_world_iterations import beside_idle, constant

pytestmark = pytest.mark.gpu


def test_gradient_where_the_forward_keeps_no_snapshots(gpu):
    """One segment of snapshots beyond what a forward keeps: the backward replays it itself. The
    oracle's gradient, and that of shorter segments, which are kept."""
    sc = beside_idle(scenes.tower(2, 2, 3, seed=4))
    n, iterations = sc.n_bodies, sc.params.iterations
    limit = constant("avbd_adjoint.cuh", "LAST_SEGMENT_BYTES")
    step_bytes = 32 * n * (5 + 2 * (iterations + 1)) + 8 * iterations * n * constant("avbd_adjoint.cuh", "LDL_STRIDE")
    steps = limit // step_bytes + 1
    target = _target(sc)
    _, loss, whole, *_ = _gpu_gradient(sc, steps, steps, target)
    _, loss2, parts, *_ = _gpu_gradient(sc, steps, 4, target)
    ref = _reference(sc, steps)
    rloss, rg = ref.adj_gradient(ref.adj_theta0(), target)
    assert loss == pytest.approx(rloss, rel=1e-10) and loss2 == pytest.approx(rloss, rel=1e-10)
    # the tolerance of the other gradient tests: the same map in 64 bits, sums in another order
    for g in (whole, parts):
        assert np.linalg.norm(g - rg) <= 1e-6 * np.linalg.norm(rg)


@pytest.mark.parametrize("steps,every", [(1, 1), (6, 6), (6, 10), (8, 4), (12, 3), (11, 3)])
def test_backward_again(gpu, steps, every):
    """Backwards after one forward, with one, two and four segments and a ragged last one: each
    gives the gradient of a forward of its own (64-bit atomic sums differ in order alone), also for
    another seed in between."""
    sc = scenes.tower(3, 3, 3, seed=4)
    rs = np.random.default_rng(3)
    seeds = rs.standard_normal((2, sc.n_bodies, 3))

    def fresh(seed):
        w = World(sc)
        w.adjoint_forward(steps, every)
        g = w.adjoint_backward(d_pos=seed)
        w.close()
        return g

    want = [fresh(s) for s in seeds]
    w = World(sc)
    w.adjoint_forward(steps, every)
    for which in (0, 1, 1, 0):
        got = w.adjoint_backward(d_pos=seeds[which])
        for k, v in want[which].items():
            assert np.linalg.norm(got[k] - v) <= 1e-9 * max(np.linalg.norm(v), 1e-300), k
    w.close()
