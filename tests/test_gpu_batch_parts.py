"""Batches of more than 1024 proxies per SM are solved by kernels of their own, a block for each part of
whole worlds, with more parts than SMs: the same bits as the grid-wide solve (no constraint joins two
worlds, so the order between them changes nothing), and the oracle's for some worlds.
"""
import numpy as np
import pytest

import b2g
import parity
import scenes

pytestmark = pytest.mark.gpu


def _batch(lo, hi, worlds, extra=0, seed=11):
    s = scenes.batched(num_worlds=worlds, lo=lo, hi=hi, seed=seed)
    if extra:
        # a world of its own size in front: more bodies than a block caches, in a part of its own
        big = scenes.batched(num_worlds=1, lo=extra, hi=extra, seed=seed + 1)
        b, f = s["bodies"].copy(), s["fixtures"].copy()
        b["world_index"] += 1
        f["body"] += len(big["bodies"])
        s = dict(s, bodies=np.concatenate([big["bodies"], b]), fixtures=np.concatenate([big["fixtures"], f]),
                 num_worlds=worlds + 1)
    return s


def _run(s, part_solve, steps, throw=None):
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    w.set_part_solve(part_solve)
    scenes.build_world(w, s)
    out = []
    for k in range(steps):
        if throw is not None and k in throw:
            w.set_linear_velocity(1, (0.0, throw[k]))
        w.step(s["dt"], s["vi"], s["pi"])
        out.append(w.get_body_states().tobytes())
    parts = w.get_step_stats()["parts"]
    w.close()
    return out, parts


# even worlds of a few bodies, uneven ones, and a world of 6000 bodies (of which a block caches 2048)
@pytest.mark.parametrize("lo,hi,worlds,extra", [(60, 62, 2700, 0), (16, 2048, 420, 6000)])
def test_batch_parts_match_the_grid_wide_solve(built, lo, hi, worlds, extra):
    s = _batch(lo, hi, worlds, extra)
    assert len(s["bodies"]) > 1024 * 152
    a, parts = _run(s, True, 40)
    b, none = _run(s, False, 40)
    assert parts > 152 and none == 0
    assert a == b


def test_a_partition_that_splits_a_world_is_made_again(built):
    """A body thrown fast makes the grounds no longer large beside the largest dynamic box: they move into
    their worlds' own hierarchies, and every later world's Morton ranks with them, between two partitions."""
    s = _batch(60, 62, 2700)
    throw = {30: 200.0, 34: 0.0, 37: -150.0, 38: 0.0}
    a, parts = _run(s, True, 44, throw)
    b, _ = _run(s, False, 44, throw)
    assert parts > 152 and a == b


def test_batch_parts_match_the_oracle(built, oracle_lib):
    s = _batch(16, 2048, 460)
    for r in parity.lockstep_window(s, steps=3, skip=60, worlds=[0, 7, 459]):
        assert r["hook_misses"] == 0 and r["bitexact_bodies"], r
        assert r["contact_key_mismatch"] == 0 and r["contact_id_mismatch"] == 0, r
