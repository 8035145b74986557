"""The narrowphase that lists contacts by kind (small worlds; large worlds of mixed shapes) against the one
that takes the table as it comes, which a launch configuration with a polygon group selects: the same bits.
"""
import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


def _run(s, group, steps):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s.get("num_worlds", 1))
    w.set_allow_sleeping(False)
    w.set_launch_config(collide_group=group)
    scenes.build_world(w, s)
    out = []
    for _ in range(steps):
        w.step(s["dt"], s["vi"], s["pi"])
        out.append(w.get_body_states().tobytes())
    n = w.get_counts()
    w.close()
    return out, n


# a handful of contacts, a warp's worth, several tiles of a block, the largest world of the small rule and
# the first past it; then a batch past the large one (several full tiles to a block)
@pytest.mark.parametrize("bodies", [3, 30, 130, 600, 2043, 2044])
def test_small_worlds_by_kind(built, bodies):
    s = scenes.mixed(n_circles=bodies // 2, n_polygons=bodies - bodies // 2, size=max(3.0, 0.7 * bodies ** 0.5), seed=bodies)
    a, _ = _run(s, 0, 30)
    b, _ = _run(s, 1, 30)
    assert a == b


def test_small_world_of_boxes_by_kind(built):
    a, _ = _run(scenes.pyramid(rows=20), 0, 60)
    b, _ = _run(scenes.pyramid(rows=20), 1, 60)
    assert a == b


def test_large_batch_by_kind(built):
    s = scenes.batched(num_worlds=420, lo=16, hi=2048, seed=5)
    assert len(s["bodies"]) > 1024 * 152
    a, _ = _run(s, 0, 40)
    b, _ = _run(s, 32, 40)
    assert a == b
