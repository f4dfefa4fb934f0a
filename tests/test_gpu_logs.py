"""Collision logs of the differentiation calls: their sizes, what they hold, and runs they are too small for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vx", "vy")


def start(edmd, N, seed, **kw):
    s = edmd.hex_start(N, 0.5, seed)
    s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], **kw)
    return s


def test_intervals_longer_than_any_log(edmd):
    """An interval longer than the run is the run; a capacity whose bytes no integer holds is refused."""
    s = start(edmd, 60, 3)
    res = []
    for every in (50, 2 ** 62, 2 ** 63 - 1):
        eng = edmd.Engine([s])
        assert edmd.load().edmd_set_log_capacity(eng.h, 2 ** 60) == edmd.ERR_CUDA
        _, lyap = eng.tangent(2, 50, every, seed=4)
        lyap_b = eng.tangent_batch(2, 50, every, seed=4)
        g = eng.msd_gradient(50, ckpt_every=every)
        gb = eng.msd_gradient_batch(50, ckpt_every=every)
        eng.advance(max_coll=10)
        res.append((lyap, lyap_b, *[x[1][k] for x in (g, gb) for k in KEYS], eng.state(0)["x"]))
        eng.close()
    for r in res[1:]:
        for a, b in zip(r, res[0]):
            np.testing.assert_array_equal(a, b)
