"""Worlds that step as one-cluster kernels (k_front, k_back: up to 4096 proxies) against the oracle, at the
sizes where the choice or a kernel's split changes: one block and its neighbour sizes, the largest rank
sort and the first radix sort of the proxy keys, the largest cluster world and the first world past it.
The bar is the parity tests': the same IEEE operations, so bodies bit for bit, pairs and contacts equal.
"""
import numpy as np
import pytest

import b2g
import parity
import scenes

pytestmark = pytest.mark.gpu


def _check(recs):
    for r in recs:
        assert r["hook_misses"] == 0 and r["pairs_equal"] and r["fat_aabb_equal"], r
        assert r["contact_key_mismatch"] == 0 and r["contact_id_mismatch"] == 0, r
        assert r["bitexact_bodies"], r


# a dense box of that many proxies (four of them walls), its bodies fast enough that every step makes
# hundreds to thousands of new pairs and rebuilds the hierarchy
@pytest.mark.parametrize("proxies", [5, 128, 129, 257, 2048, 2049, 4096, 4097])
def test_cluster_world_matches_the_oracle(built, oracle_lib, proxies):
    n = proxies - 4
    s = scenes.mixed(n_circles=n // 2, n_polygons=n - n // 2, size=max(6.0, 1.2 * n ** 0.5), seed=proxies)
    s["bodies"]["linear_velocity"] *= 20.0
    recs = parity.lockstep_window(s, steps=5)
    _check(recs)
    assert n < 100 or recs[-1]["constraints"] > n // 4


# one proxy alone (a hierarchy of one leaf, no contact), and a body on a ground box
@pytest.mark.parametrize("count", [1, 2])
def test_cluster_world_of_one_and_two_proxies(built, oracle_lib, count):
    s = scenes.hello_world()
    s["bodies"]["allow_sleep"] = 0
    if count == 1:
        s["bodies"], s["fixtures"] = s["bodies"][1:], s["fixtures"][1:]
        s["fixtures"]["body"] = 0
    _check(parity.lockstep_window(s, steps=90))


# a resting world: the hierarchy is kept between passes and most steps have no new pair
def test_cluster_world_at_rest_matches_the_oracle(built, oracle_lib):
    recs = parity.lockstep_window(scenes.pyramid(rows=12), steps=40, skip=60)
    _check(recs)
    assert recs[-1]["constraints"] > 100


def test_profile_phases_follow_each_other(built):
    """The phase times of a cluster world and of a larger one: none negative, their sum is the step."""
    for n in (200, 6000):
        s = scenes.mixed(n_circles=n // 2, n_polygons=n // 2, size=1.5 * n ** 0.5)
        w = b2g.B2world(gravity=s["gravity"])
        w.set_allow_sleeping(False)
        scenes.build_world(w, s)
        for _ in range(4):
            w.step(s["dt"], s["vi"], s["pi"])
            t, p = w.get_phase_times(tree_split=True), w.get_profile()
            assert all(v >= 0.0 for v in t.values()) and t["solver"] > 0.0, t
            assert abs(sum(t[k] for k in w.PHASES) - p["step"]) < 1e-3, (t, p)
        w.close()
