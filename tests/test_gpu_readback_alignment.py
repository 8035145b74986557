"""Body states read back into arrays at any address, waited for or not: those that the device's stores cannot take
go by way of a copy. The same states, and nothing written around them."""
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


@pytest.mark.parametrize("wait", [True, False])
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 6, 8, 12, 13])
def test_any_address(world, wait, offset):
    whole = world.get_body_states()
    for count in (1, 257, 790):
        raw = np.full(32 * count + 64, 0xA5, np.uint8)
        start = (-raw.ctypes.data) % 16 + 16 + offset
        out = raw[start:start + 32 * count].view(b2g.BODY_STATE)
        if wait:
            world.get_body_states(first=9, count=count, out=out)
        else:
            for _ in range(3):  # both device buffers, and one of them again
                world.get_body_states_async(out, first=9)
            world.wait_body_states()
        assert out.tobytes() == whole[9:9 + count].tobytes()
        assert np.all(raw[:start] == 0xA5) and np.all(raw[start + 32 * count:] == 0xA5)
