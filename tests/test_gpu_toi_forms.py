"""b2g_time_of_impact reads the caller's arrays in place and builds the shapes on the device: the counts
at which a block's piece of the arrays ends, arrays off their type's alignment (which go by way of a
copy), every way to define a polygon, and a definition of no shape, against the oracle bit for bit."""
import numpy as np
import pytest

import b2g
import oracle
import test_toi

pytestmark = pytest.mark.gpu


def _off(a):
    """The same items at an address one byte past a multiple of 8."""
    raw = np.zeros(a.nbytes + 16, np.uint8)
    start = (-raw.ctypes.data) % 8 + 1
    view = raw[start:start + a.nbytes].view(a.dtype)
    view[:] = a
    return view


def _pairs(n, seed=23):
    da, sa, db, sb = test_toi._random_pairs(n, seed)
    rng = np.random.default_rng(seed)
    for k in range(0, n, 4):  # boxes, turned boxes and vertex lists the hull gives up on or welds
        d = da if k % 8 else db
        d[k] = b2g.box_fixture(0, float(rng.uniform(0.05, 0.5)), float(rng.uniform(0.05, 0.5)))
        if k % 3 == 0:
            d[k]["polygon_mode"] = b2g.POLYGON_BOX_ORIENTED
            d[k]["box_center"] = rng.uniform(-0.3, 0.3, 2)
            d[k]["box_angle"] = rng.uniform(-3, 3)
        if k % 5 == 0:
            d[k]["polygon_mode"] = b2g.POLYGON_HULL
            d[k]["vertex_count"] = k % 11
            d[k]["vertices"] = rng.uniform(-0.4, 0.4, (8, 2)) if k % 2 == 0 else 0.25
    return da, sa, db, sb


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("aligned", [True, False])
def test_counts_and_alignment_match_the_oracle(built, oracle_lib, n, aligned):
    arrays = _pairs(n)
    t_max = np.random.default_rng(n).uniform(0.2, 1.0, n).astype(np.float32)
    oracle.set_trig(False)  # the project's sin/cos, which the GPU uses
    try:
        ref = oracle.time_of_impact(*arrays, t_max)
    finally:
        oracle.set_trig(True)
    got = b2g.time_of_impact(*(arrays if aligned else map(_off, arrays)), t_max)
    assert np.array_equal(got["state"], ref["state"])
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))


@pytest.mark.parametrize("kind", [-1, 3, 1 << 20])
def test_no_shape_is_refused_and_nothing_written(built, kind):
    lib = b2g.load_library()
    da, sa, db, sb = _pairs(300)
    db["shape_type"][299] = kind
    out = np.full(300, 7, b2g.TOI_OUTPUT)
    before = out.copy()
    rc = lib.b2g_time_of_impact(b2g._ptr(da), b2g._ptr(sa), b2g._ptr(db), b2g._ptr(sb), None, 300, b2g._ptr(out))
    assert rc == b2g.ERR_INVALID_ARG
    assert np.array_equal(out, before)
