"""Every row of the sin/cos table (b2g_trig_table.h) is sin(j/512) and cos(j/512) as a float and the float of what
is left, from their Taylor series in 60-digit arithmetic; and the rows cover the reduced range."""
import math
import os
import re
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _f32(x):
    """The float nearest to a Decimal: from the double nearest to it, checked against its neighbours."""
    near = np.float32(float(x))
    cands = [near, np.nextafter(near, np.float32(np.inf)), np.nextafter(near, np.float32(-np.inf))]
    exact = Fraction(x)
    return min(cands, key=lambda f: abs(Fraction(float(f)) - exact))


def test_rows():
    getcontext().prec = 60
    text = open(os.path.join(ROOT, "box2d-rs_gb300", "csrc", "b2g_trig_table.h")).read()
    text = re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)
    values = [float.fromhex(t.rstrip("f")) if "0x" in t else float(t.rstrip("f")) for t in re.findall(r"[-+0-9a-fxp.]+f", text)]
    rows = np.array(values).reshape(-1, 4)
    assert len(rows) == 403
    assert round(512 * math.pi / 4) == 402  # the last row is the nearest of j/512 to pi/4
    for j, row in enumerate(rows):
        x = Decimal(j) / 512
        term, s, c = Decimal(1), Decimal(0), Decimal(0)
        for k in range(60):
            if k % 2:
                s += term if k % 4 == 1 else -term
            else:
                c += term if k % 4 == 0 else -term
            term = term * x / (k + 1)
        for value, hi, lo in ((s, row[0], row[1]), (c, row[2], row[3])):
            assert np.float32(hi) == hi and np.float32(lo) == lo
            assert hi == _f32(value), j
            assert lo == _f32(value - Decimal(float(hi))), j
