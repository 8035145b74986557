"""Worlds that may sleep through both forms of the narrowphase, at the sizes where one takes over from the other
and where a step leaves its cluster: stacks at rest fall asleep, and a ball that reaches them then wakes one
after another, chains of wakes within one pass among them. The same bits in both forms, and the oracle's."""
import numpy as np
import pytest

import b2g
import parity
import scenes

pytestmark = pytest.mark.gpu


def _stacks(n, seed=7):
    """A ground, n bodies in stacks of three (two boxes and a circle or a box) 0.62 m apart, and a heavy ball that
    gravity does not pull, which flies along them from step 90 on."""
    rng = np.random.default_rng(seed)
    bodies = b2g.body_defs(n + 2)
    bodies["allow_sleep"] = 1
    bodies["type"] = b2g.DYNAMIC
    bodies[0]["type"] = b2g.STATIC
    i = np.arange(n)
    cols = -(-n // 3)
    bodies["position"][2:, 0] = 0.62 * (i // 3) + rng.uniform(-0.01, 0.01, n)
    bodies["position"][2:, 1] = 0.26 + 0.52 * (i % 3)
    bodies["position"][1] = (-68.0, 0.9)
    bodies["linear_velocity"][1] = (45.0, 0.0)
    bodies["gravity_scale"][1] = 0.0
    fixtures = b2g.fixture_defs(n + 2)
    fixtures["body"] = np.arange(n + 2)
    fixtures["friction"] = 0.6
    fixtures["density"] = 1.0
    fixtures["shape_type"] = b2g.POLYGON
    fixtures["polygon_mode"] = b2g.POLYGON_BOX
    fixtures["box_half_extents"] = (0.25, 0.25)
    fixtures["box_half_extents"][2:, 0] = rng.uniform(0.22, 0.26, n)
    fixtures["shape_type"][0] = b2g.EDGE
    fixtures["vertices"][0, 1], fixtures["vertices"][0, 2] = (-50.0, 0.0), (0.62 * cols + 50.0, 0.0)
    round_ = np.concatenate([[False, True], (i % 6 == 5)])
    fixtures["shape_type"][round_] = b2g.CIRCLE
    fixtures["radius"][round_] = 0.25
    fixtures["radius"][1] = 0.5
    fixtures["density"][1] = 20.0
    return {"bodies": bodies, "fixtures": fixtures, "gravity": (0.0, -10.0), "dt": np.float32(1.0 / 60.0), "vi": 8, "pi": 3,
            "num_worlds": 1, "allow_sleep": True}


STEPS, ARRIVES = 150, 90


def _run(s, group):
    w = b2g.B2world(gravity=s["gravity"])
    w.set_allow_sleeping(True)
    w.set_launch_config(collide_group=group)
    scenes.build_world(w, s)
    out, awake = [], []
    for _ in range(STEPS):
        w.step(s["dt"], s["vi"], s["pi"])
        a = w.get_awake()
        out.append(w.get_body_states().tobytes() + a.tobytes())
        awake.append(int(a.sum()))
    w.close()
    return out, awake


# proxies: one stack, a few, the largest of the small rule and the next, the largest cluster and the next
@pytest.mark.parametrize("n", [3, 120, 2046, 2047, 4094, 4095])
def test_sleeping_stacks_in_both_forms(built, n):
    s = _stacks(n)
    a, awake = _run(s, 0)
    assert min(awake[ARRIVES - 5:ARRIVES]) < n // 4 + 2  # most have fallen asleep
    assert awake[-1] > min(awake[ARRIVES - 5:ARRIVES])   # and some were woken
    assert a == _run(s, 1)[0]


@pytest.mark.parametrize("n", [3, 2046, 4095])
def test_sleeping_stacks_lockstep(built, n):
    recs, _, _ = parity.lockstep(_stacks(n), STEPS, check_pairs=False, check_contacts=False)
    for r in recs:
        assert r["hook_misses"] == 0 and r["bitexact_bodies"] and r["awake_equal"], r
    assert min(r["awake"] for r in recs) < n // 4 + 2
