"""Large batches: a kept partition that has split a world is made afresh, and only then. The count of them is read
from the counters in a saved state."""
import ctypes
import struct

import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu

COUNTERS, PART_REMADE = 64, 63  # 32-bit counters of a world, and the one asked for


def _sms():
    rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
    n = ctypes.c_int(0)
    assert rt.cudaDeviceGetAttribute(ctypes.byref(n), 16, 0) == 0  # cudaDevAttrMultiProcessorCount
    return n.value


def _remade(w):
    state = bytes(w.save_state())
    n_alloc = struct.unpack_from("<i", state, 48)[0]
    sizes = struct.unpack_from(f"<{n_alloc}Q", state, 120)
    at = [i for i, b in enumerate(sizes) if b == 4 * COUNTERS]
    assert len(at) == 1
    start = 120 + 8 * n_alloc + sum(sizes[:at[0]])
    return np.frombuffer(state, np.int32, COUNTERS, start)[PART_REMADE]


@pytest.mark.parametrize("kinematic", [False, True])
def test_partitions_made_again(built, kinematic):
    s = scenes.batched(num_worlds=2700, lo=60, hi=62, seed=11)
    ground = np.nonzero(s["bodies"]["type"] == b2g.STATIC)[0]
    if kinematic:
        s["bodies"]["type"][ground + 2] = b2g.KINEMATIC
    w = b2g.B2world(gravity=s["gravity"], num_worlds=s["num_worlds"])
    w.set_allow_sleeping(False)
    scenes.build_world(w, s)
    assert w.get_counts()["fixtures"] > 1024 * _sms()
    for _ in range(30):
        w.step(s["dt"], s["vi"], s["pi"])
    assert w.get_step_stats()["parts"] > _sms() and _remade(w) == 0
    # a body thrown fast: the grounds are no longer large beside the largest dynamic box, move into their
    # worlds' own hierarchies and back, and every later world's Morton ranks with them
    throw = {0: 200.0, 4: 0.0, 7: -150.0, 8: 0.0}
    for k in range(14):
        if k in throw:
            w.set_linear_velocity(1, (0.0, throw[k]))
        w.step(s["dt"], s["vi"], s["pi"])
    assert _remade(w) >= 1
    w.close()
