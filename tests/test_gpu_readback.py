"""b2g_get_body_states at the counts where a block's piece ends, from an odd first body, into arrays on a
16-byte boundary and off it: the same states as the whole read, and nothing written around them."""
import numpy as np
import pytest

import b2g
import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(built):
    s = scenes.mixed(n_circles=400, n_polygons=400, size=30.0, seed=3)
    w = b2g.B2world(gravity=s["gravity"])
    scenes.build_world(w, s)
    for _ in range(3):
        w.step(s["dt"], s["vi"], s["pi"])
    yield w
    w.close()


@pytest.mark.parametrize("count", [1, 255, 256, 257, 770])
@pytest.mark.parametrize("offset", [0, 4, 8, 12])
def test_ranges_and_alignment(world, count, offset):
    whole = world.get_body_states()
    raw = np.full(32 * count + 64, 0xA5, np.uint8)
    start = (-raw.ctypes.data) % 16 + 16 + offset
    out = raw[start:start + 32 * count].view(b2g.BODY_STATE)
    world.get_body_states(first=7, count=count, out=out)
    assert out.tobytes() == whole[7:7 + count].tobytes()
    assert np.all(raw[:start] == 0xA5) and np.all(raw[start + 32 * count:] == 0xA5)
