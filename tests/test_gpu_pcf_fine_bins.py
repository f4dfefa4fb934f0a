"""g(r) with bins far below single precision's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 1e-21: squared distances below 2^-126; 1e-200: their squares are no numbers; 1e-11 and 1e-13: both sides of the rule
@pytest.mark.parametrize("dr", [1e-11, 1e-13, 1e-21, 1e-200])
def test_points_close_together(edmd, oracle, dr):
    rng = np.random.default_rng(4)
    n, side = 60, 24.0
    # points (radius zero) around the corner of the box; the positions are sums of a few bins, so FP64 holds them
    x, y = rng.integers(0, 40, n) * dr, rng.integers(0, 40, n) * dr
    s = dict(x=x, y=y, vx=np.zeros(n), vy=np.zeros(n), rad=np.zeros(n), m=np.ones(n), type=np.ones(n, np.int32), N=n,
             vr=None, desc=edmd.default_desc(n, side, side))
    eng = edmd.Engine([s])
    o = oracle.Oracle(arrays={k: s[k] for k in ("x", "y", "vx", "vy", "rad", "m", "type")}, Lx=side, Ly=side)
    r, g = eng.pcf(0, dr, 30.5 * dr)
    ro, go = o.pcf(dr, 30.5 * dr)
    eng.close()
    np.testing.assert_array_equal(r, ro)
    np.testing.assert_array_equal(g, go)
    assert dr < 1e-150 or (g > 0).sum() > 15
