"""Boxes of one or two cells along an axis, where the 3x3 scan visits a cell more than once.

The crossing times of such boxes are only sound while nothing moves across the
narrow axis (the nearest image of a cell's wall can lie behind the disk, in the
reference as well), so the disks move along the long one: a chain of unequal
masses.  Every call bounds its events.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vx", "vy")
ALL = KEYS + ("rad", "m")


def chain(edmd, narrow, turned, m2, cells=9, n=16):
    """n disks in a row in a box of `cells` x `narrow` cells (turned: the other way round)."""
    rng = np.random.default_rng(narrow + 5)
    L, W = 2.0 * cells + 0.3, 2.0 * narrow + 0.7
    along, v = (np.arange(n) + 0.5) * L / n, rng.standard_normal(n)
    across, still, m = np.full(n, 0.8 * W), np.zeros(n), np.ones(n)
    m[::2] = m2
    s = dict(x=along, y=across, vx=v, vy=still, Lx=L, Ly=W)
    if turned:
        s = dict(x=across, y=along, vx=still, vy=v, Lx=W, Ly=L)
    s.update(rad=np.full(n, 0.3), m=m, type=np.ones(n, np.int32), N=n, vr=None)
    s["desc"] = edmd.default_desc(n, s["Lx"], s["Ly"])
    return s


@pytest.mark.parametrize("narrow,turned,m2", [(1, False, 1.0), (1, True, 0.51), (2, False, 0.51), (2, True, 1.0), (3, False, 0.51)])
def test_chain_against_the_oracle(edmd, oracle, narrow, turned, m2):
    import torch
    s = chain(edmd, narrow, turned, m2)
    o = oracle.Oracle(arrays={k: s[k] for k in ALL + ("type",)}, Lx=s["Lx"], Ly=s["Ly"])
    _, n = o.run(400, cap=1)
    assert n == 400
    o.sync()
    ost, t = o.state(), o.t
    eng = edmd.Engine([s])
    eng.advance(max_coll=400, max_events=20000)
    eng.sync()
    st, c = eng.state(0), eng.counters(0)
    eng.close()
    for k in KEYS:
        np.testing.assert_array_equal(st[k], ost[k], err_msg=k)
    oc = o.counters()
    assert {k: c[k] for k in oc} == oc and c["t"] == t
    # the allocation-free entry point (its events are bounded by itself)
    L = edmd.load()
    bufs = {k: torch.tensor(s[k], dtype=torch.float64, device="cuda:0") for k in ALL}
    torch.cuda.synchronize()
    ncol, tout = C.c_int64(), C.c_double()
    rc = L.edmd_run_noalloc(C.byref(s["desc"]), *[C.c_void_p(bufs[k].data_ptr()) for k in ALL], 400, float("inf"),
                            C.byref(ncol), C.byref(tout), None)
    assert rc == edmd.OK, L.edmd_last_error(None)
    for k in KEYS:
        np.testing.assert_array_equal(bufs[k].cpu().numpy(), ost[k], err_msg=k)
    assert ncol.value == 400 and tout.value == t


@pytest.mark.parametrize("narrow,turned", [(1, False), (2, True)])
def test_growing_chain_as_with_16_lanes(edmd, narrow, turned):
    res = []
    for lanes in (16, 32):
        s = chain(edmd, narrow, turned, 0.51)
        s["vr"] = np.full(s["N"], 0.02)
        s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], vr_base=0.1, dtime=0.7, dtime_thermo=0.9)
        edmd.set_warp_group(lanes)
        try:
            eng = edmd.Engine([s, chain(edmd, 4, False, 0.51)])
            for k in range(1, 8):
                eng.advance(max_coll=20 * k, max_events=20000)
            eng.sync()
            res.append((eng.states(), eng.all_counters(), eng.thermo(0)))
            eng.close()
        finally:
            edmd.set_warp_group(32)
    for k in KEYS:
        np.testing.assert_array_equal(res[0][0][k], res[1][0][k], err_msg=k)
    for k, v in res[0][1].items():
        np.testing.assert_array_equal(v, res[1][1][k], err_msg=k)
    np.testing.assert_array_equal(res[0][2], res[1][2])


@pytest.mark.parametrize("ny,seed", [(2, 1), (2, 2), (5, 3)])
def test_collisions_across_the_border_of_two_cells(edmd, oracle, ny, seed):
    """Eight disks around a corner of four cells, for as long as none leaves its cell."""
    rng = np.random.default_rng(seed)
    Lx, Ly = 4.9, 2.0 * ny + 0.7
    dx = np.array([-1, 1, -1, 1, -1, 1, -1, 1]) * 0.36
    dy = np.array([-1, -1, 1, 1, -3, -3, 3, 3]) * 0.34
    v = rng.normal(0, 0.2, (2, 8))
    s = dict(x=Lx / 2 + dx, y=Ly / ny + dy, vx=v[0] - 2 * dx, vy=v[1] - dy, rad=np.full(8, 0.3),
             m=np.where(np.arange(8) % 3, 0.51, 1.0), type=np.ones(8, np.int32), N=8, vr=None,
             desc=edmd.default_desc(8, Lx, Ly))
    o = oracle.Oracle(arrays={k: s[k] for k in ALL + ("type",)}, Lx=Lx, Ly=Ly)
    _, n = o.run(12, cap=1)
    o.sync()
    oc, ost = o.counters(), o.state()
    assert n == 12 and oc["ncross"] == 0
    eng = edmd.Engine([s])
    eng.advance(max_coll=12, max_events=200)
    eng.sync()
    st, c = eng.state(0), eng.counters(0)
    eng.close()
    for k in KEYS:
        np.testing.assert_array_equal(st[k], ost[k], err_msg=k)
    assert {k: c[k] for k in oc} == oc and c["t"] == o.t
