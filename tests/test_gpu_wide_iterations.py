"""The wide iteration kernel (avbd_iterate_flow.cuh) at the edges of its groups, rounds and
chunks, bit for bit against the CPU oracle; at the edge of its body count against the
per-colour launches, which share none of its data flow."""
import math
import os
import re

import numpy as np
import pytest

from avbd_demo3d_b200 import World, scenes
from test_gpu_parity import assert_same_state, lockstep

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avbd_demo3d_b200", "csrc")


def params(**kw):
    return scenes.baseline_params(**kw)


def plate(side, iterations=10):
    """A slab carrying side^2 small boxes: 4 side^2 + 4 contact rows on one body."""
    b = scenes.SceneBuilder(f"plate{side}", params(iterations=iterations))
    b.body((60, 60, 1), 0.0, 0.5, (0, 0, -0.5))
    b.body((side * 1.2, side * 1.2, 0.5), 1.0, 0.6, (0, 0, 0.25))
    for i in range(side * side):
        x, y = (i % side - (side - 1) / 2) * 1.1, (i // side - (side - 1) / 2) * 1.1
        b.body((0.8, 0.9, 0.7), 1.0, 0.5, (x, y, 0.85))
    return b.build()


def hub(arms, iterations=10, fracture=math.inf):
    """A box jointed to `arms` others (3 rows each, angular parts on every second one), springs
    between neighbours, one arm anchored to the world, and two overlapping static boxes."""
    b = scenes.SceneBuilder(f"hub{arms}", params(iterations=iterations))
    b.body((80, 80, 1), 0.0, 0.5, (0, 0, -0.5))
    b.body((1, 1, 1), 0.0, 0.5, (20, 0, 0.4))  # rests in the ground: contacts without a dynamic body
    c = b.body((2, 2, 1), 1.0, 0.5, (0, 0, 4))
    ids = []
    for k in range(arms):
        a = 2 * math.pi * k / arms
        r = 3.0 + 1.5 * (k % 3)
        d = b.body((0.5, 0.4, 0.3), 1.0 + 0.1 * k, 0.5, (r * math.cos(a), r * math.sin(a), 4.0 + 0.05 * k))
        b.joint(c, d, (0.5 * r * math.cos(a), 0.5 * r * math.sin(a), 0), (-0.5 * r * math.cos(a), -0.5 * r * math.sin(a), 0),
                math.inf, (50.0 if fracture == math.inf else math.inf) if k % 2 else 0.0, fracture)
        ids.append(d)
    for k in range(0, arms - 1, 3):
        b.spring(ids[k], ids[k + 1], (0, 0, 0.1), (0, 0, -0.1), 200.0, 1.0)
    b.joint(None, ids[0], (3, 0, 5), (0, 0, 0.15))
    return b.build()


CASES = {
    "rows_1": lambda: plate(1),
    "rows_20": lambda: plate(2),
    "rows_40_two_rounds": lambda: plate(3),
    "rows_148": lambda: plate(6),
    "one_iteration": lambda: plate(3, iterations=1),
    "joints_2": lambda: hub(2),
    "joints_11_across_rounds": lambda: hub(11),
    "joints_37": lambda: hub(37, iterations=7),
    "joints_two_iterations": lambda: hub(9, iterations=2),
    "joints_break": lambda: hub(12, fracture=40.0),
    "round_bodies": lambda: scenes.round_mix(50, seed=5, cols=3),
    "more_chunks_than_warps": lambda: scenes.stack_grid(25, 25, 12, seed=9),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_wide_iterations_match_oracle(gpu, name):
    lockstep(CASES[name](), 3 if name == "more_chunks_than_warps" else 25)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,height", [(19, 503, 3), (28, 64, 16)])  # 28,672 and 28,673 bodies
def test_both_sides_of_the_body_limit(gpu, nx, ny, height):
    scene = scenes.stack_grid(nx, ny, height, seed=3)
    a, b = World(scene), World(scene)
    b.set_iteration_mode(0)
    for s in range(3):
        a.step(1)
        b.step(1)
    assert_same_state(a, b, scene.name)
    a.close()
    b.close()


def test_stick_threshold_is_the_root_test():
    """x < STICK_THRESH_SQ is sqrtf(x) < 1e-5f for every float: both are monotone in x, and they
    turn at the same float."""
    text = open(os.path.join(CSRC, "avbd_kernels.cuh")).read()
    limit = np.float32(float.fromhex(re.search(r"STICK_THRESH_SQ = (0x[0-9a-fp.+-]+)f;", text).group(1)))
    thresh = np.float32(0.00001)
    below = np.nextafter(limit, np.float32(0), dtype=np.float32)
    assert np.sqrt(below) < thresh and not np.sqrt(limit) < thresh
