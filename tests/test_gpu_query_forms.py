"""World queries at the counts where their kernels split the work, against the oracle: boxes in and past a
block's eight, lists that are empty, longer than the lists a warp keeps (256), longer than the device
sorts (1024) and of every fixture; capacities that are exact and one too small; arrays off their type's
alignment (which go by way of a copy) and worlds of a batch that do not exist."""
import ctypes

import numpy as np
import pytest

import b2g
import parity
import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def worlds(built):
    s = scenes.mixed(n_circles=2500, n_polygons=2500, size=75.0, seed=41)
    recs, gpu, ora = parity.lockstep(s, 6, check_pairs=False, check_contacts=False)
    assert recs[-1]["bitexact_bodies"] and recs[-1]["fat_aabb_equal"]
    yield gpu, ora
    gpu.close()


def _boxes(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-5.0, 80.0, (n, 2))
    e = rng.uniform(0.05, 2.0, (n, 2))
    e[::5] *= 6.0      # some of hundreds of fixtures
    e[3::50] *= 12.0   # and of more than a thousand
    b = np.concatenate([c - e, c + e], 1)
    if n > 6:
        b[2] = (-100.0, -100.0, 200.0, 200.0)  # every fixture
        b[5] = (300.0, 300.0, 301.0, 301.0)    # none
    return b.astype(np.float32)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 600])
def test_boxes_match_the_oracle(worlds, n):
    gpu, ora = worlds
    boxes = _boxes(n, n)
    q = gpu.query_aabb(boxes)
    assert np.array_equal(q, ora.query_aabb(boxes))
    if n == 600:
        counts = np.bincount(q[:, 0], minlength=n)
        assert counts[5] == 0 and counts[2] == 5004
        assert ((counts > 256) & (counts <= 1024)).any() and ((counts > 1024) & (counts < 5004)).any()


def _raw(gpu, boxes, out, capacity):
    n = ctypes.c_int32(-1)
    rc = gpu._lib.b2g_query_aabb(gpu._h, b2g._ptr(boxes), None, len(boxes), b2g._ptr(out), capacity, ctypes.byref(n))
    return rc, n.value


def test_capacity_exact_and_one_too_small(worlds):
    gpu, ora = worlds
    boxes = _boxes(40, 3)
    ref = ora.query_aabb(boxes)
    out = np.full((len(ref), 2), 77, np.uint32)
    rc, n = _raw(gpu, boxes, out, len(ref) - 1)
    assert rc == b2g.ERR_CAPACITY and n == len(ref) and np.all(out == 77)
    rc, n = _raw(gpu, boxes, out, len(ref))
    assert rc == b2g.OK and n == len(ref) and np.array_equal(out, ref)


def _off(a):
    raw = np.zeros(a.nbytes + 16, np.uint8)
    start = (-raw.ctypes.data) % 4 + 1
    view = raw[start:start + a.nbytes].view(a.dtype).reshape(a.shape)
    view[...] = a
    return view


def test_misaligned_arrays_give_the_same(worlds):
    gpu, _ = worlds
    boxes = _boxes(60, 5)
    ref = gpu.query_aabb(boxes)
    out = _off(np.zeros((len(ref), 2), np.uint32))
    rc, n = _raw(gpu, _off(boxes), out, len(ref))
    assert rc == b2g.OK and n == len(ref) and np.array_equal(out, ref)
    rays = np.random.default_rng(2).uniform(-5.0, 80.0, (777, 4)).astype(np.float32)
    hits = gpu.ray_cast_closest(rays)
    out = _off(np.zeros(len(rays), b2g.RAY_HIT))
    r = _off(rays)
    assert gpu._lib.b2g_ray_cast_closest(gpu._h, b2g._ptr(r), None, len(r), b2g._ptr(out)) == b2g.OK
    assert out.tobytes() == hits.tobytes() and (hits["fixture"] >= 0).sum() > 300


def test_queries_of_a_world_that_is_not_there(built):
    s = scenes.batched(num_worlds=3, lo=16, hi=32, seed=2)
    w = b2g.B2world(gravity=s["gravity"], num_worlds=3)
    scenes.build_world(w, s)
    w.step(s["dt"], s["vi"], s["pi"])
    boxes = np.tile(np.array([[-50.0, -50.0, 50.0, 50.0]], np.float32), (4, 1))
    q = w.query_aabb(boxes, np.array([0, 3, 2, 4000], np.uint32))
    assert set(q[:, 0]) == {0, 2}
    hits = w.ray_cast_closest(np.tile(np.array([[0.0, 20.0, 0.0, -5.0]], np.float32), (2, 1)), np.array([1, 3], np.uint32))
    assert hits["fixture"][0] >= 0 and hits["fixture"][1] == -1
    w.close()
