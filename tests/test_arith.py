"""Integer-pipe division and square root (csrc/edmd_arith.cuh) against IEEE FP64, on the host.

The header compiles as host C++ with the FP32 seeds moved by a given number of
units in the last place, so the tolerance of the digits is tested too.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r"""
#include "edmd_arith.cuh"
extern "C" void div_all(const double* a, const double* b, double* q, unsigned char* other, long n, int ulps) {
  for (long i = 0; i < n; i++) { bool o; q[i] = edmd::div_normal(a[i], b[i], &o, ulps); other[i] = o; }
}
extern "C" void sqrt_all(const double* x, double* s, unsigned char* other, long n, int ulps) {
  for (long i = 0; i < n; i++) { bool o; s[i] = edmd::sqrt_normal(x[i], &o, ulps); other[i] = o; }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("arith")
    (d / "a.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", str(d / "a.so"), str(d / "a.cpp"),
                    "-I" + os.path.join(ROOT, "graphical-edmd_gb300", "csrc")], check=True)
    return ctypes.CDLL(str(d / "a.so"))


def p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def operands(n=200000):
    rng = np.random.default_rng(11)
    bits = rng.integers(0, 1 << 64, (2, n), dtype=np.uint64)
    keep = rng.integers(0, 53, n).astype(np.uint64)
    tail = (np.uint64(1) << keep) - np.uint64(1)
    a, b = bits[0].copy(), bits[1].copy()
    a[: n // 4] &= ~tail[: n // 4]                            # short significands: exact quotients and roots
    b[n // 8: n // 3] |= tail[n // 8: n // 3]                 # long runs of ones
    near = slice(n // 2, 3 * n // 4)                          # nearly equal significands, ordinary exponents
    m = np.uint64((1 << 52) - 1)
    b[near] = (b[near] & ~m) | ((a[near] + rng.integers(0, 5, n // 4).astype(np.uint64) - np.uint64(2)) & m)
    e = rng.integers(900, 1150, (2, n)).astype(np.uint64) << np.uint64(52)
    half = slice(n // 3, n)
    a[half] = (a[half] & (m | np.uint64(1 << 63))) | e[0][half]
    b[half] = (b[half] & (m | np.uint64(1 << 63))) | e[1][half]
    edge = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, np.nextafter(2.0 ** -1022, 0),
                     np.nextafter(np.inf, 0), 1 + 2.0 ** -52, 2 - 2.0 ** -52, 0.5])
    x, y = (g.ravel() for g in np.meshgrid(edge, edge))
    return np.concatenate([a.view(np.float64), x]), np.concatenate([b.view(np.float64), y])


@pytest.mark.parametrize("ulps", [0, -8, 8])
def test_quotients_and_roots_equal_ieee_bit_for_bit(lib, ulps):
    a, b = operands()
    with np.errstate(all="ignore"):
        q, s = a / b, np.sqrt(np.abs(a))
    got, other = np.empty_like(a), np.empty(len(a), np.uint8)
    lib.div_all(p(a), p(b), p(got), p(other), ctypes.c_long(len(a)), ulps)
    normal = lambda v: np.isfinite(v) & (np.abs(v) >= 2.0 ** -1022)  # noqa: E731
    own = other == 0
    assert np.array_equal(got[own].view(np.uint64), q[own].view(np.uint64))
    # everything the digits hand over has an operand or a result that is not an ordinary normal number
    assert not np.any(other[normal(a) & normal(b) & normal(q) & (np.abs(q) > 2.0 ** -1021)])
    assert own.sum() > len(a) // 2
    x = np.abs(a)
    # squares and their neighbours
    t = np.sqrt(x[normal(x)])
    t = (t.view(np.uint64) & ~np.uint64((1 << 26) - 1)).view(np.float64)
    sq = (t * t).view(np.uint64)
    x = np.concatenate([x, sq.view(np.float64), (sq - np.uint64(1)).view(np.float64), (sq + np.uint64(1)).view(np.float64), -x[:100]])
    got, other = np.empty_like(x), np.empty(len(x), np.uint8)
    lib.sqrt_all(p(x), p(got), p(other), ctypes.c_long(len(x)), ulps)
    own = other == 0
    with np.errstate(all="ignore"):
        s = np.sqrt(x)
    assert np.array_equal(got[own].view(np.uint64), s[own].view(np.uint64))
    assert np.array_equal(own, normal(x) & (x > 0))


WALK = r"""
#include "edmd_arith.cuh"
extern "C" void walk_both(double d, double tc, double* P, unsigned long* k) {
  uint64_t n = k[1];
  for (int i = 0; i < (1 << 24) && P[0] + d <= tc; i++) { P[0] += d; k[0]++; }
  edmd::walk_calendar(d, tc, P[1], n);
  k[1] = n;
}
"""


def test_calendar_walk_equals_repeated_additions(tmp_path):
    (tmp_path / "w.cpp").write_text(WALK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", str(tmp_path / "w.so"), str(tmp_path / "w.cpp"),
                    "-I" + os.path.join(ROOT, "graphical-edmd_gb300", "csrc")], check=True)
    w = ctypes.CDLL(str(tmp_path / "w.so"))
    rng = np.random.default_rng(5)
    for n in range(600):
        N = int(rng.integers(2, 3000 if n % 3 else 2000000))
        d = 5.0 / N if n % 7 else np.ldexp(1.0 + rng.integers(0, 4), -int(rng.integers(0, 30)))      # widths that tie too
        P0 = 0.0 if n % 2 else float(np.add.accumulate(np.full(int(rng.integers(1, 50000)), d))[-1])
        if n % 11 == 0:
            P0 = np.ldexp(1.0 + rng.random(), int(rng.integers(-10, 50)))                            # steps below half an ulp among them
        tc = P0 + rng.random() * d * (100000 if n % 5 == 0 else 3000) if n % 13 else P0 - 1.0
        P = np.array([P0, P0])
        k = np.array([7, 7], np.uint64)
        w.walk_both(ctypes.c_double(d), ctypes.c_double(tc), p(P), p(k))
        assert P[0] == P[1] and k[0] == k[1], (d, tc, P0)
