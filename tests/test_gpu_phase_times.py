"""Phase times of a step whose broadphase pass the host repeats with grown capacities: those of the step's own
passes, without the host's work in between."""
import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [800, 5000])  # on a cluster and on the grid
def test_phases_of_a_step_that_grows(built, n):
    s = scenes.pile(n_boxes=n, width=24.0, height=60.0, seed=3, spacing=0.6)
    w = b2g.B2world(gravity=s["gravity"], contact_capacity=64, pair_capacity=64)
    w.set_allow_sleeping(False)
    w.set_auto_grow(True)
    scenes.build_world(w, s)
    grown, other, grows = [], [], 0
    for k in range(160):
        w.step(s["dt"], s["vi"], s["pi"])
        t, now = w.get_phase_times(), w.get_step_stats()["capacity_grows"]
        assert all(v >= 0.0 for v in t.values())
        if k >= 3:  # the first launches of a process load the kernels
            (grown if now > grows else other).append(t["solver"])
        grows = now
    w.close()
    assert len(grown) >= 1 and len(other) >= 100
    assert max(grown) <= 3.0 * max(other), (max(grown), max(other))
