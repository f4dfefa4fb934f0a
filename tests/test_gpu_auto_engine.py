"""EDMD_ENGINE_AUTO: the engine that a context reports is the one that runs it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vx", "vy")


def starts(edmd):
    out = []
    for k in range(3):
        s = edmd.hex_start(12 + 2 * k, 0.5, k + 1)
        s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], tmax=1e9)
        out.append(s)
    return out


# both sides of the line between the engines, and where it was before
@pytest.mark.parametrize("nsys,lane", [(3, False), (16384, False), (28671, False), (28672, True)])
def test_auto_reports_what_runs(edmd, nsys, lane):
    one = starts(edmd)
    ref = []
    for s in one:
        e = edmd.Engine([s], engine=edmd.ENGINE_WARP)
        e.advance(max_coll=120)
        e.sync()
        ref.append((e.state(0), e.counters(0)))
        e.close()
    eng = edmd.Engine([one[k % 3] for k in range(nsys)])
    assert eng.engine == (edmd.ENGINE_LANE if lane else edmd.ENGINE_WARP)
    eng.advance(max_coll=120)
    if lane:
        assert eng.last_launches() == 1                   # no table of waiting systems
    eng.sync()
    st, cnt = eng.states(), eng.all_counters()
    off = np.cumsum([0] + eng.N)
    for s in range(nsys):
        r = ref[s % 3]
        for k in KEYS:
            assert np.array_equal(st[k][off[s]:off[s + 1]], r[0][k]), (s, k)
    for k in ("ncol", "ncross", "nstale", "npair", "t"):
        np.testing.assert_array_equal(cnt[k], np.resize([r[1][k] for r in ref], nsys), err_msg=k)
    # the differentiation calls run where the warp engine is reported, and are refused where it is not
    if lane:
        with pytest.raises(edmd.EngineError):
            eng.msd_gradient_batch(10)
    else:
        msd, g = eng.msd_gradient_batch(10)
        assert msd.shape == (nsys,) and np.isfinite(g["vx"]).all()
        for s in (0, nsys - 1):
            e = edmd.Engine([one[s % 3]])
            e.advance(max_coll=120)
            m1, g1 = e.msd_gradient(10)
            e.close()
            # the batched form adds a system's displacements over a tree
            np.testing.assert_allclose(msd[s], m1, rtol=1e-12)
            for k in KEYS:
                np.testing.assert_allclose(g[k][off[s]:off[s + 1]], g1[k], rtol=1e-9, atol=1e-9 * np.abs(g1[k]).max())
    eng.close()
