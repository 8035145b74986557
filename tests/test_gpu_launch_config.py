"""The launch configuration that a world reports is the one it runs with: writing it back changes nothing, 0
solver threads means by the world's size, and the autotuner spends no steps on knobs that nothing reads."""
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


def _world(s, steps=3):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    scenes.build_world(w, s)
    for _ in range(steps):
        w.step(s["dt"], s["vi"], s["pi"])
    return w


# a batch past one cluster's size, one world past it, and one on a cluster
@pytest.mark.parametrize("scene,threads", [
    (lambda: scenes.batched(num_worlds=20, lo=250, hi=251, seed=4), 512),
    (lambda: scenes.mixed(n_circles=2500, n_polygons=2500, size=75.0, seed=41), 256),
    (lambda: scenes.mixed(n_circles=300, n_polygons=300, size=25.0, seed=41), 256)])
def test_reported_solver_block_is_the_one_that_runs(built, scene, threads):
    s = scene()
    w = _world(s)
    c = w.get_launch_config()
    assert c["solver_block"] == threads
    w.set_launch_config(**c)
    assert w.get_launch_config() == c
    w.set_launch_config(**dict(c, solver_block=512))
    assert w.get_launch_config()["solver_block"] == 512
    w.set_launch_config(**dict(c, solver_block=0))
    assert w.get_launch_config() == c
    w.step(s["dt"], s["vi"], s["pi"])
    w.set_part_solve(False)
    w.step(s["dt"], s["vi"], s["pi"])
    w.close()


def test_autotune_leaves_knobs_that_a_small_world_does_not_read(built):
    s = scenes.mixed(n_circles=40, n_polygons=40, size=12.0, seed=5)
    w = _world(s)
    before = w.get_launch_config()
    cfg = w.autotune(s["dt"], s["vi"], s["pi"], 2)
    # the narrowphase's two knobs, three candidates each of two untimed and two timed steps
    assert w.tuning_steps() == 2 * 3 * 4
    for knob in ("coop_blocks_per_sm", "traverse_block", "solver_block"):
        assert cfg[knob] == before[knob]
    w.close()
