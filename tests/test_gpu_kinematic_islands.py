"""Bodies that touch nothing but one kinematic body are one island, over as many parts of the part-local solve
as the bodies lie in, and no constraint between two parts says so: the early exit of the position iterations
waits for all of them. Against the oracle step by step, and the same bits in a second run."""
import numpy as np
import pytest

import b2g
import parity
import scenes

pytestmark = pytest.mark.gpu


def _slab(n, seed=3):
    """n bodies 0.6 m apart dropped from up to 0.3 m onto one kinematic slab that moves sideways; they never
    meet."""
    rng = np.random.default_rng(seed)
    bodies = b2g.body_defs(n + 1)
    bodies["allow_sleep"] = 0
    bodies["type"] = b2g.DYNAMIC
    bodies[0]["type"] = b2g.KINEMATIC
    bodies[0]["linear_velocity"] = (0.05, 0.0)
    x = (np.arange(n) - 0.5 * (n - 1)) * 0.6
    bodies[1:]["position"][:, 0] = x
    bodies[1:]["position"][:, 1] = 0.65 + rng.uniform(0.0, 0.3, n)
    fixtures = b2g.fixture_defs(n + 1)
    fixtures["body"] = np.arange(n + 1)
    fixtures["shape_type"] = b2g.POLYGON
    fixtures["polygon_mode"] = b2g.POLYGON_BOX
    fixtures["density"] = 1.0
    fixtures["friction"] = 0.5
    fixtures["box_half_extents"][0] = (0.3 * n + 5.0, 0.5)
    fixtures["box_half_extents"][1:] = rng.uniform(0.08, 0.15, (n, 2))
    round_ = np.arange(n + 1) % 3 == 1
    fixtures["shape_type"][round_] = b2g.CIRCLE
    fixtures["radius"][round_] = 0.12
    return {"bodies": bodies, "fixtures": fixtures, "gravity": (0.0, -10.0), "dt": np.float32(1.0 / 60.0), "vi": 8, "pi": 3,
            "num_worlds": 1, "allow_sleep": False}


def _states(s, steps, part_solve=True, throw=None):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    w.set_part_solve(part_solve)
    scenes.build_world(w, s)
    out, stats = [], []
    for k in range(steps):
        if throw is not None and k in throw:
            w.set_linear_velocity(throw["body"], (0.0, throw[k]))
        w.step(s["dt"], s["vi"], s["pi"])
        out.append(w.get_body_states().tobytes())
        stats.append(w.get_step_stats())
    w.close()
    return out, stats


# two parts and the largest world of one cluster; the smallest of the grid-wide kernels and a larger one
@pytest.mark.parametrize("n", [600, 4095, 4096, 9001])
def test_bodies_on_one_kinematic_slab_lockstep(built, n):
    s = _slab(n)
    recs, gpu, _ = parity.lockstep(s, 40)
    for r in recs:
        assert r["hook_misses"] == 0 and r["bitexact_bodies"], r
    stats = gpu.get_step_stats()
    assert stats["parts"] > 1 and stats["colours"] == 0 and stats["interior_slots"] >= n
    a, st = _states(s, 40)
    assert any(x["parts"] > 1 and x["colours"] == 0 and x["constraints"] > 0 for x in st)
    assert a == _states(s, 40)[0]


def _batch_on_kinematic(worlds, per):
    """Worlds of bodies over a static ground, a body of each turned into a kinematic one in their midst."""
    s = scenes.batched(num_worlds=worlds, lo=per, hi=per, seed=19)
    ground = np.nonzero(s["bodies"]["type"] == b2g.STATIC)[0]
    s["bodies"]["type"][ground + 2] = b2g.KINEMATIC
    return s, ground


@pytest.mark.parametrize("worlds", [30, 60])  # on one cluster and on the grid
def test_batch_with_kinematic_bodies_lockstep(built, worlds):
    s, _ = _batch_on_kinematic(worlds, 100)
    recs, gpu, _ = parity.lockstep(dict(s, allow_sleep=False), 60)
    for r in recs:
        assert r["hook_misses"] == 0 and r["bitexact_bodies"], r
    assert gpu.get_step_stats()["parts"] > 1


def test_large_batch_with_kinematic_bodies_over_a_partition_made_again(built):
    """More parts than SMs, whose solver has no barrier to take: a kept partition that no longer holds each
    world in one part is made afresh (a body thrown fast moves the grounds into their worlds' hierarchies
    and all ranks after them), here with a kinematic body in every world."""
    s, ground = _batch_on_kinematic(2700, 61)
    throw = {"body": int(ground[0]) + 1, 30: 200.0, 34: 0.0, 37: -150.0, 38: 0.0}
    a, st = _states(s, 44, True, throw)
    assert st[-1]["parts"] > 152
    b, _ = _states(s, 44, False, throw)
    assert a == b
