"""A dense box query's buffers are given back when the call returns; those of ordinary ones stay with the world."""
import ctypes

import numpy as np
import pytest

import b2g

pytestmark = pytest.mark.gpu


def _free():
    rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
    free, total = ctypes.c_size_t(0), ctypes.c_size_t(0)
    assert rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_a_dense_query_leaves_no_large_buffer(built):
    n, m = 20_000, 1500
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
    few = w.query_aabb(boxes[:2])
    before = _free()
    out = np.zeros((n * m, 2), np.uint32)
    count = ctypes.c_int32(0)
    rc = w._lib.b2g_query_aabb(w._h, b2g._ptr(boxes), None, m, b2g._ptr(out), len(out), ctypes.byref(count))
    assert rc == b2g.OK and count.value == n * m  # 120 MB of lists
    assert np.array_equal(out[:, 0], np.repeat(np.arange(m), n)) and np.array_equal(out[:n, 1], np.arange(n))
    assert _free() >= before - (32 << 20)
    assert np.array_equal(w.query_aabb(boxes[:2]), few)
    w.close()
