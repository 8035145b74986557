"""The broadphase's sorts at the sizes where their split changes: the last rank count and the first radix
sort of the whole grid, one, two and several rows of 256 keys to a tile, and a cluster's radix sort; each
against the oracle: equal pairs, contacts in the same order, bodies bit for bit."""
import pytest

import parity
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("proxies", [2049, 2304, 8192, 8193, 38912, 38913, 90001])
def test_sorts_match_the_oracle(built, oracle_lib, proxies):
    n = proxies - 4
    s = scenes.mixed(n_circles=n // 2, n_polygons=n - n // 2, size=1.1 * n ** 0.5, seed=proxies)
    s["pair_capacity"] = s["contact_capacity"] = 64 * n
    s["bodies"]["linear_velocity"] *= 8.0
    for r in parity.lockstep_window(s, steps=3):
        assert r["hook_misses"] == 0 and r["pairs_equal"] and r["fat_aabb_equal"], r
        assert r["contact_key_mismatch"] == 0 and r["contact_id_mismatch"] == 0, r
        assert r["bitexact_bodies"], r
