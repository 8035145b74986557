"""The continuous pass finds a moved proxy's new pairs by a warp's walk of the hierarchies: worlds whose
hierarchy is a single leaf, a few leaves, and one that puts more nodes on the walk's pending list than a
round takes, against the oracle. The bar is the parity tests': bodies bit for bit, contacts equal."""
import numpy as np
import pytest

import b2g
import parity

pytestmark = pytest.mark.gpu


# a disc at 110 m/s in a box of thin walls, over a grid of small circles at rest of which every 16th collides
# with it: with 3600 of them its fat box covers thousands of leaves
@pytest.mark.parametrize("circles", [0, 1, 31, 3600])
def test_fast_disc_over_circles(built, oracle_lib, circles):
    bodies = b2g.body_defs(circles + 2)
    bodies["allow_sleep"] = 0
    bodies[1:]["type"] = b2g.DYNAMIC
    bodies[1]["position"] = (3.0, 2.9)
    bodies[1]["linear_velocity"] = (80.0, 75.0)
    k = np.arange(circles)
    bodies["position"][2:, 0] = 0.4 + (k % 60) * 0.12
    bodies["position"][2:, 1] = 0.4 + (k // 60) * 0.12
    fx = [b2g.edge_fixture(0, a, b, restitution=1.0, friction=0.0) for a, b in
          (((0.0, 0.0), (8.0, 0.0)), ((8.0, 0.0), (8.0, 8.0)), ((8.0, 8.0), (0.0, 8.0)), ((0.0, 8.0), (0.0, 0.0)))]
    fx += [b2g.circle_fixture(1, 0.3, density=50.0, restitution=1.0, friction=0.0)]
    fx += [b2g.circle_fixture(int(i) + 2, 0.04, density=1.0) for i in k]
    fx = np.concatenate(fx)
    fx["group_index"][4:] = -1
    fx["group_index"][5::16] = 0
    s = {"name": "disc", "bodies": bodies, "fixtures": fx, "gravity": (0.0, 0.0),
         "dt": np.float32(1.0 / 60.0), "vi": 8, "pi": 3, "steps": 25, "num_worlds": 1, "allow_sleep": False,
         "n_dynamic": circles + 1, "continuous": True}
    recs, gpu, ora = parity.lockstep(s, 25, check_pairs=False)
    for r in recs:
        assert r["hook_misses"] == 0 and r["bitexact_bodies"], r
        assert r["contact_key_mismatch"] == 0 and r["contact_id_mismatch"] == 0, r
    events = gpu.get_toi_stats()[0]
    assert events == ora.toi_events() and events > 5
