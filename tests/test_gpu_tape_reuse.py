"""A tape of the sizes of the one before takes over its buffers: the gradient is a fresh world's, whatever the
last tape held (the same steps, more of them, steps that an edit made invalid, a tape never ended)."""
import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


def _world(s):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    scenes.build_world(w, s)
    for _ in range(25):
        w.step(s["dt"], s["vi"], s["pi"])
    return w


def _gradient(w, s, start, steps, max_steps=12, interval=5):
    w.load_state(start)
    w.tape_begin(max_steps, interval)
    for _ in range(steps):
        w.step(s["dt"], s["vi"], s["pi"])
    w.tape_end()
    info = w.tape_info()
    assert info["valid"] and info["steps"] == steps
    d = np.zeros(w.body_count, b2g.BODY_STATE)
    d["world_center"] = np.random.default_rng(5).normal(size=(w.body_count, 2))
    g = w.backward(d)
    assert w.tape_info()["replay_mismatches"] == 0
    return g[s["bodies"]["type"] == b2g.DYNAMIC]


@pytest.mark.parametrize("before", ["same", "longer", "invalid", "unended", "other_sizes"])
def test_second_tape_is_a_first_one(built, before):
    s = scenes.throw_stack_batch(seeds=3)
    fresh = _world(s)
    start = fresh.save_state()
    expected = _gradient(fresh, s, start, 7)
    fresh.close()
    w = _world(s)
    if before == "invalid":
        w.tape_begin(12, 5)
        w.step(s["dt"], s["vi"], s["pi"])
        w.set_linear_velocity(int(s["projectiles"][0]), (1.0, 2.0))
        w.step(s["dt"], s["vi"], s["pi"])
        w.tape_end()
        assert not w.tape_info()["valid"]
    elif before == "unended":
        w.tape_begin(12, 5)
        w.step(s["dt"], s["vi"], s["pi"])
        w.tape_begin(12, 5)
        w.tape_end()
    elif before == "other_sizes":
        _gradient(w, s, start, 7, max_steps=9, interval=4)
    else:
        _gradient(w, s, start, 7 if before == "same" else 12)
    got = _gradient(w, s, start, 7)
    w.close()
    for f in b2g.BODY_STATE.names:
        assert np.array_equal(got[f], expected[f]), f
