"""The backward pass at the sizes where its launches change (one block, clusters of blocks, a cooperative
grid) and with its segments replayed side by side: steps that fill their last segment, leave one step over
or fit one segment, and tapes with as many segments as steps. The replay lands on the recorded states, and a
tape cut into other segments gives the same gradient but for rounding in the shared bodies' sums."""
import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


def _gradient(s, steps, interval, part_solve=True, skip=25):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    w.set_part_solve(part_solve)
    scenes.build_world(w, s)
    for _ in range(skip):
        w.step(s["dt"], s["vi"], s["pi"])
    w.tape_begin(steps, interval)
    for _ in range(steps):
        w.step(s["dt"], s["vi"], s["pi"])
    w.tape_end()
    d = np.zeros(w.body_count, b2g.BODY_STATE)
    d["world_center"] = np.random.default_rng(5).normal(size=(w.body_count, 2))
    g, again = w.backward(d), w.backward(d)
    info = w.tape_info()
    w.close()
    assert info["replay_mismatches"] == 0 and info["steps"] == steps
    dyn = s["bodies"]["type"] == b2g.DYNAMIC
    for f in b2g.BODY_STATE.names:  # no atomics on dynamic bodies but the carried impulses' sums of one term
        assert np.array_equal(g[f][dyn], again[f][dyn]), f
    return g[dyn]


# one block; two to sixteen; past the clusters' slots
@pytest.mark.parametrize("worlds", [1, 9, 40, 130])
def test_segments_do_not_change_the_gradient(built, worlds):
    s = scenes.throw_stack_batch(seeds=worlds)
    whole = _gradient(s, 17, 17)
    assert np.isfinite(whole["linear_velocity"]).all() and np.abs(whole["linear_velocity"]).max() > 0.0
    for interval in (16, 4, 1):
        g = _gradient(s, 17, interval)
        for f in b2g.BODY_STATE.names:
            assert np.array_equal(g[f], whole[f]), (interval, f)


def test_grid_wide_colours(built):
    """Without the part-local solve every colour is a boundary colour of the tape."""
    s = scenes.throw_stack_batch(seeds=3)
    a, b = _gradient(s, 12, 12, part_solve=False), _gradient(s, 12, 5, part_solve=False)
    for f in b2g.BODY_STATE.names:
        assert np.array_equal(a[f], b[f]), f
