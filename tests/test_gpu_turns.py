"""More systems than lane groups: systems of different length take turns, every one as when it runs alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vx", "vy")
COUNTS = ("ncol", "ncross", "nstale", "npair", "npred", "nevents", "t", "stop_reason")


# 3040 groups of 32 lanes are resident, 4864 of 16, 19456 of 4; a turn is 256 events (1024 for a call of at most
# 256 collisions), and the systems below take 20 to 2000, so that some end while others still change places
@pytest.mark.parametrize("lanes,nsys", [(32, 3041), (32, 3100), (32, 7000), (16, 5000), (4, 20000)])
def test_systems_in_turns_equal_single_systems(edmd, oracle, lanes, nsys):
    starts = []
    for k, tmax in enumerate((1e9, 0.3, 4.0, 1e9, 9.0, 1e9, 1.5)):
        s = edmd.hex_start(34 + 12 * k, 0.5, k + 1)
        s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], tmax=tmax)
        starts.append(s)
    calls = (900, 200, 300)
    ref = []
    for s in starts:
        eng = edmd.Engine([s])
        for c in calls:
            eng.advance(max_coll=c)
        eng.sync()
        ref.append((eng.state(0), eng.counters(0)))
        eng.close()
    assert {r[1]["stop_reason"] for r in ref} == {1, 3} and max(r[1]["nevents"] for r in ref) > 1800
    o = oracle.Oracle(arrays={k: starts[3][k] for k in KEYS + ("rad", "m", "type")}, Lx=starts[3]["Lx"], Ly=starts[3]["Ly"])
    o.run(sum(calls), cap=1)
    o.sync()
    ost = o.state()
    order = np.random.default_rng(nsys).integers(0, len(starts), nsys)
    edmd.set_warp_group(lanes)
    try:
        eng = edmd.Engine([starts[k] for k in order], engine=edmd.ENGINE_WARP)
        for c in calls:
            eng.advance(max_coll=c)
            assert eng.last_launches() == 2               # the table of waiting systems, the event loop
        eng.sync()
        st, cnt = eng.states(), eng.all_counters()
        eng.close()
    finally:
        edmd.set_warp_group(32)
    for k in KEYS:
        np.testing.assert_array_equal(ref[3][0][k], ost[k], err_msg=k)
        np.testing.assert_array_equal(st[k], np.concatenate([ref[q][0][k] for q in order]), err_msg=k)
    for k in COUNTS:
        np.testing.assert_array_equal(cnt[k], [ref[q][1][k] for q in order], err_msg=k)
