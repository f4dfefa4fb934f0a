"""Sizes at which the kernels' splits can go wrong: every engine against the serial algorithm, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EXACT = 32
KEYS = ("x", "y", "vx", "vy")


def start(edmd, N, phi, seed, **kw):
    s = edmd.hex_start(N, phi, seed)
    s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], **kw)
    return s


def oracle_state(oracle, s, coll=None, t_stop=None):
    o = oracle.Oracle(arrays={k: s[k] for k in ("x", "y", "vx", "vy", "rad", "m", "type")}, Lx=s["Lx"], Ly=s["Ly"])
    if coll is not None:
        _, n = o.run(coll, cap=1)
    else:
        _, n = o.run(10 ** 12, t_stop=t_stop, cap=1)
    o.sync()
    return o.state(), n


def same(a, b):
    for k in KEYS:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# leaves 32 (two levels), 1023 / 1024 / 1025 + 3 specials (three or four levels), 2049 (chunks of 4096 initial
# events), 16383 / 16385 (host or device check of a staged state)
@pytest.mark.parametrize("N", [29, 1020, 1022, 2049, 16383, 16390])
def test_start_states_at_the_splits_of_the_set_up(edmd, oracle, N):
    s = start(edmd, N, 0.60, 7)
    eng = edmd.Engine([s])
    eng.load_state(*[s[k] for k in ("x", "y", "vx", "vy", "rad", "m")])
    eng.advance(max_coll=400)
    eng.sync()
    ost, _ = oracle_state(oracle, s, coll=400)
    same(eng.state(0), ost)
    eng.close()


@pytest.mark.parametrize("per_cell", [7, 8, 20])
def test_crowded_cells(edmd, oracle, per_cell):
    """Small disks, many to a cell: candidate lists at and past their buffers, in the serial and the round engine."""
    rng = np.random.default_rng(per_cell)
    side, n = 12.0, 36 * per_cell
    g = int(np.ceil(np.sqrt(n)))
    pos = rng.permutation(g * g)[:n]
    s = dict(x=(pos % g + 0.5) * side / g, y=(pos // g + 0.5) * side / g, vx=rng.standard_normal(n), vy=rng.standard_normal(n),
             rad=np.full(n, 0.04), m=np.ones(n), type=np.ones(n, np.int32), N=n, Lx=side, Ly=side)
    s["desc"] = edmd.default_desc(n, side, side)
    eng = edmd.Engine([s])
    eng.advance(max_coll=300)
    eng.sync()
    ost, _ = oracle_state(oracle, s, coll=300)
    same(eng.state(0), ost)
    t = eng.counters(0)["t"]
    eng.load_state(*[s[k] for k in ("x", "y", "vx", "vy", "rad", "m")])
    eng.advance_rounds(t_stop=t / 2, radius=3, flags=EXACT)
    eng.sync()
    rst = eng.state(0)
    eng.load_state(*[s[k] for k in ("x", "y", "vx", "vy", "rad", "m")])
    eng.advance(t_stop=t / 2)
    eng.sync()
    same(rst, eng.state(0))
    eng.close()


# number of systems around one warp per SM sub-partition, one block of four warps at three per SM, and the five-block build
@pytest.mark.parametrize("nsys", [3, 610, 1216, 1217, 1830, 3100])
def test_batch_sizes_share_one_result(edmd, oracle, nsys):
    starts = [start(edmd, 40 + 2 * (k % 5), 0.5, k % 5 + 1) for k in range(5)]
    eng = edmd.Engine([starts[k % 5] for k in range(nsys)])
    eng.advance(max_coll=150)
    eng.sync()
    st = eng.states()
    off = np.cumsum([0] + eng.N)
    for q in range(5):
        if q >= nsys:
            continue
        ost, _ = oracle_state(oracle, starts[q], coll=150)
        for s in {q, q + 5 * ((nsys - 1 - q) // 5)}:
            for k in KEYS:
                np.testing.assert_array_equal(st[k][off[s]:off[s + 1]], ost[k])
    eng.close()


# 20 disks: a tree of two levels and a box of few cells; 29 / 30: two and three levels; 200: cells of their own
@pytest.mark.parametrize("N,additive", [(20, False), (29, False), (30, True), (200, False), (200, True)])
def test_two_warps_equal_one(edmd, N, additive):
    """Few systems have two warps each: growth, samples, calendar wraps and stops of every kind as with 16 lanes."""
    kw = dict(tmax=1e9, dtime=0.4, dtime_thermo=0.3, contact=edmd.CONTACT_ADDITIVE if additive else edmd.CONTACT_NONADDITIVE)
    res = []
    for lanes in (16, 32):
        s = edmd.grow_start(N, 0.45, 11)
        s["desc"] = edmd.default_desc(s["N"], s["Lx"], s["Ly"], vr_base=s["vr_base"], **kw)
        edmd.set_warp_group(lanes)
        try:
            eng = edmd.Engine([s, s])
            for k in range(1, 30):
                eng.advance(max_coll=k * 7 if k % 3 else 2 ** 62, t_stop=1.7 * k if k % 3 == 0 else float("inf"))
            eng.sync()
            c = {k: v for k, v in eng.counters(1).items()}
            res.append((eng.state(1), c, eng.thermo(1)))
            eng.close()
        finally:
            edmd.set_warp_group(32)
    same(res[0][0], res[1][0])
    assert res[0][1] == res[1][1]
    np.testing.assert_array_equal(res[0][2], res[1][2])


@pytest.mark.parametrize("energy,t0,t1", [(1.0, 0.0, 0.02), (1.0, 70.0, 70.6), (1e6, 0.0, 0.0006), (1e-6, 3000.0, 3100.0)])
def test_round_selection_at_other_time_scales(edmd, energy, t0, t1):
    """The selection's 32-bit times: early and late in a run, fast and slow systems."""
    s = start(edmd, 600, 0.55, 3, tmax=1e9)
    v = np.sqrt(energy)
    s["vx"], s["vy"] = s["vx"] * v, s["vy"] * v
    args = [s[k] for k in ("x", "y", "vx", "vy", "rad", "m")]
    a, b = edmd.Engine([s]), edmd.Engine([s])
    if t0 > 0:
        a.advance_rounds(t_stop=t0, radius=4, flags=EXACT)
        b.advance(t_stop=t0)
    a.advance_rounds(t_stop=t1, radius=4, flags=EXACT)
    b.advance(t_stop=t1)
    assert a.counters(0)["ncol"] == b.counters(0)["ncol"] and len(args) == 6
    a.sync()
    b.sync()
    same(a.state(0), b.state(0))
    a.close()
    b.close()


# one lane, both row-register builds at their edges, all columns; qr_every leaves an odd and an even number of chunks
@pytest.mark.parametrize("K,n_coll", [(1, 60), (16, 100), (17, 80), (32, 100)])
def test_tangent_batch_equals_single_systems(edmd, K, n_coll):
    starts = [start(edmd, N, 0.60, 2) for N in (33, 120, 200)]
    eng = edmd.Engine(starts)
    lyap = eng.tangent_batch(K, n_coll, 20, seed=5)
    eng.close()
    for s, st in enumerate(starts):
        one = edmd.Engine([st])
        _, ref = one.tangent(K, n_coll, 20, seed=5 + s)
        assert len(one.log(0)) == 20                      # the last chunk's collisions
        one.close()
        # the two forms add a Gram matrix's rows in another order: 2 QRs of 20 collisions each, condition ~1e3
        np.testing.assert_allclose(lyap[s], ref, rtol=1e-9, atol=1e-9 * np.abs(ref).max())


def test_gradient_of_a_run_too_long_for_one_log(edmd):
    """4096 systems x 8300 collisions exceed the log kept for a whole call: the checkpointed sweep, against single systems."""
    starts = [start(edmd, 12 + 2 * (k % 3), 0.5, k % 3 + 1, tmax=1e9) for k in range(3)]
    eng = edmd.Engine([starts[k % 3] for k in range(4096)])
    msd, g = eng.msd_gradient_batch(8300, ckpt_every=4150)
    off = np.cumsum([0] + eng.N)
    eng.close()
    for s in range(3):
        one = edmd.Engine([starts[s]])
        m1, g1 = one.msd_gradient(8300, ckpt_every=1000)
        one.close()
        for q in (s, s + 3 * 1364):
            a, b = off[q], off[q + 1]
            np.testing.assert_allclose(msd[q], m1, rtol=1e-12)
            for k in ("vx", "vy", "x", "y"):
                np.testing.assert_allclose(g[k][a:b], g1[k], rtol=1e-9, atol=1e-9 * np.abs(g1[k]).max())


# wide and narrow bins (lattice distances fall on their edges at the start), a reach that is no multiple of the bin
@pytest.mark.parametrize("dr,max_r,coll", [(0.5, 6.0, 0), (3.0, 7.7, 0), (0.004, 12.0, 2000), (0.05, 9.99, 2000)])
def test_pcf_bins(edmd, oracle, dr, max_r, coll):
    s = start(edmd, 3000, 0.60, 9)
    eng = edmd.Engine([s])
    o = oracle.Oracle(arrays={k: s[k] for k in ("x", "y", "vx", "vy", "rad", "m", "type")}, Lx=s["Lx"], Ly=s["Ly"])
    if coll:
        eng.advance(max_coll=coll)
        eng.sync()
        o.run(coll, cap=1)
        o.sync()
    for _ in range(2):                                    # the second call reuses the workspace
        r, g = eng.pcf(0, dr, max_r)
        ro, go = o.pcf(dr, max_r)
        np.testing.assert_array_equal(r, ro)
        np.testing.assert_array_equal(g, go)
    eng.close()
