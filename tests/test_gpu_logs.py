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


def test_chunks_whose_logs_have_no_room_for_two(edmd):
    """One log of 1.7e11 bytes fits the GPU, two of them do not: chunks one after the other (the runs end at tmax, soon)."""
    s = start(edmd, 60, 3, tmax=3.0)
    for batch in (False, True):
        res = []
        for every, most in ((10 ** 6, 2 * 10 ** 6), (3 * 10 ** 9, 6 * 10 ** 9)):
            eng = edmd.Engine([s])
            lyap = eng.tangent_batch(3, most, every, seed=4)[0] if batch else eng.tangent(3, most, every, seed=4)[1]
            res.append((lyap, eng.counters(0)["ncol"]))
            eng.close()
        assert res[0][1] == res[1][1] > 100
        np.testing.assert_array_equal(res[0][0], res[1][0])


def crowd_out(leave):
    """Takes the GPU's memory up to `leave` bytes (given back with the returned tensor)."""
    import torch
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda:0")


@pytest.mark.parametrize("batch", [False, True])
def test_one_log_gives_the_exponents_of_two(edmd, batch):
    """340 MB of log a chunk, and 500 MB left: every chunk's log is read before the next chunk writes it."""
    import torch
    s = [start(edmd, 60 + 20 * (k % 3), 3 + k % 3) for k in range(2000)]
    res = []
    for full in (False, True):
        eng = edmd.Engine(s)
        hog = crowd_out(500 << 20) if full else None
        try:
            res.append(eng.tangent_batch(2, 10000, 3000, seed=4) if batch else eng.tangent(2, 10000, 3000, seed=4, s=7)[1])
        finally:
            del hog
            torch.cuda.empty_cache()
        n = len(eng.log(7))
        assert n == 1000                                  # the last chunk's collisions
        eng.close()
    np.testing.assert_array_equal(res[0], res[1])


@pytest.mark.parametrize("batch", [False, True])
def test_a_run_that_fails_leaves_its_last_chunk(edmd, batch):
    """Two disks meet at t = 0.05 (the first chunk); the collision at t = 0.1 finds an overlap (the second)."""
    from conftest import line_overlap_state
    s = line_overlap_state(edmd)
    s["x"][4], s["vx"][3], s["vx"][4] = 4.05, 1.0, 0.0
    s["vy"][3] = s["vy"][4] = 0.0
    eng = edmd.Engine([s])
    with pytest.raises(edmd.EngineError) as e:
        eng.tangent_batch(1, 5, 1, seed=2) if batch else eng.tangent(1, 5, 1, seed=2)
    assert e.value.code == edmd.ERR_OVERLAP
    log = eng.log(0)
    eng.close()
    assert len(log) == 1 and {int(log["i"][0]), int(log["j"][0])} == {1, 2}
    assert abs(log["t"][0] - 0.1) < 1e-12


def same_gradient(a, b):
    np.testing.assert_array_equal(a[0], b[0])
    for k in KEYS:
        np.testing.assert_array_equal(a[1][k], b[1][k], err_msg=k)


@pytest.mark.parametrize("batch", [False, True])
def test_long_intervals_bound_a_gradients_memory(edmd, batch):
    """64 systems x 19000 collisions (68 MB of log): in five segments, whose log and checkpoints take half of that, and as one."""
    import torch
    s = [start(edmd, 200, 3 + k % 2) for k in range(64)]
    res, took = [], []
    for every in (3800, 100):
        eng = edmd.Engine(s)
        eng.tangent_batch(1, 4, 2)                        # (kernels loaded, second stream made)
        free = torch.cuda.mem_get_info()[0]
        res.append(eng.msd_gradient_batch(19000, ckpt_every=every) if batch else eng.msd_gradient(19000, ckpt_every=every, s=5))
        took.append(free - torch.cuda.mem_get_info()[0])
        res[-1] += (eng.state(5),)
        eng.close()
    same_gradient(res[0], res[1])
    assert np.isfinite(res[0][1]["vx"]).all() and np.abs(res[0][1]["vx"]).max() > 0
    for k in KEYS:
        np.testing.assert_array_equal(res[0][2][k], res[1][2][k])
    assert took[0] < 45 << 20 and took[1] > 55 << 20, took


@pytest.mark.parametrize("batch", [False, True])
def test_a_gradient_without_room_for_its_log(edmd, batch):
    """230 MB of log asked for and 130 MB left: the segments' checkpoints are there already, and the result is the same."""
    import torch
    s = [start(edmd, 100, 3 + k % 2) for k in range(1024)]
    res = []
    for full in (False, True):
        eng = edmd.Engine(s)
        for k in range(22):
            eng.checkpoint_save(k)
        eng.msd_gradient_batch(2, ckpt_every=1)           # (kernels loaded)
        hog = crowd_out(130 << 20) if full else None
        try:
            res.append(eng.msd_gradient_batch(4000, ckpt_every=200) if batch else eng.msd_gradient(4000, ckpt_every=200, s=5))
        finally:
            del hog
            torch.cuda.empty_cache()
        eng.close()
    same_gradient(res[0], res[1])
