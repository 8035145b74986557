"""More overlaps than 31 bits count: the boxes' total is kept in 64 bits, the call reports that it is past the
capacity, and nothing is written."""
import ctypes

import numpy as np
import pytest

import b2g

pytestmark = pytest.mark.gpu


def test_a_total_past_31_bits(built):
    n, m = 20_000, 110_000
    bodies = b2g.body_defs(n)
    bodies["type"] = b2g.DYNAMIC
    bodies["position"][:, 0], bodies["position"][:, 1] = np.arange(n) % 150, np.arange(n) // 150
    fixtures = b2g.fixture_defs(n)
    fixtures["body"] = np.arange(n)
    fixtures["shape_type"] = b2g.CIRCLE
    fixtures["radius"] = 0.2
    w = b2g.B2world(gravity=(0.0, 0.0))
    w.create_bodies(bodies)
    w.create_fixtures(fixtures)
    w.step(1.0 / 60.0, 8, 3)
    boxes = np.tile(np.array([[-10.0, -10.0, 400.0, 400.0]], np.float32), (m, 1))
    assert n * m > 2**31
    out = np.full((64, 2), 77, np.uint32)
    count = ctypes.c_int32(-1)
    rc = w._lib.b2g_query_aabb(w._h, b2g._ptr(boxes), None, m, b2g._ptr(out), len(out), ctypes.byref(count))
    assert rc == b2g.ERR_CAPACITY and count.value == 2**31 - 1
    assert np.all(out == 77)
    few = w.query_aabb(boxes[:3])
    assert np.array_equal(few[:, 0], np.repeat(np.arange(3), n)) and np.array_equal(few[:n, 1], np.arange(n))
    w.close()
