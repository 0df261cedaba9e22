"""The step kernels' own arithmetic (csrc/rp_arith.cuh) against IEEE 754 on the host, bit for bit.

Roots, quotients and conversions stand for the library's, which round correctly
(numpy's do too), so the parity form needs the same last bit: besides random
operands over all exponents they are tried on the operands whose exact result
lies closest to a rounding boundary, built with integers:

* quotients: a 2^53 - b m = +-1, +-3, ... for an odd 54-bit m puts a / b within
  2^-53 of the midpoint m / 2^53 (in units of its last place);
* reciprocals of a root s: s m = 2^106 - r for an odd m and a small r;
* roots: (M + 1/2)^2 = M^2 + M + 1/4, so the 53-bit numbers M^2 + M + j with a
  small even j are the ones whose root lies next to a midpoint.

Comparisons stand for the floating ones, which are false for a NaN of either sign.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
U = np.uint64


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from rusty_particles_gb300 import build as b
    so = str(tmp_path_factory.mktemp("arith") / "probe.so")
    subprocess.run([b.nvcc(), *b.ARCH, *b.COMMON, *b.EXTRA["k_step.cu"], "-shared", "-cudart", "static", "-o", so,
                    os.path.join(HERE, "arith_probe.cu")], check=True, capture_output=True)
    L = ctypes.CDLL(so)
    dp = ctypes.POINTER(ctypes.c_double)
    L.probe.argtypes = [ctypes.c_int, ctypes.c_size_t, dp, dp, dp]

    def run(op, a, b=None):
        a = np.ascontiguousarray(a).view(np.float64)
        b = a if b is None else np.ascontiguousarray(b).view(np.float64)
        out = np.empty(len(a))
        assert L.probe(op, len(a), a.ctypes.data_as(dp), b.ctypes.data_as(dp), out.ctypes.data_as(dp)) == 0
        return out

    return run


def _bits(x):
    return np.ascontiguousarray(x).view(U)


def _same(got, want, *operands):
    nan = np.isnan(want)
    bad = np.where(nan, ~np.isnan(got), _bits(got) != _bits(want))
    assert not bad.any(), [(int(bad.sum()), len(bad))] + [tuple(float(o[i]).hex() for o in (*operands, got, want))
                                                          for i in np.flatnonzero(bad)[:4]]


def _doubles(rng, n, emin=0, emax=2047):
    """Random sign and mantissa, exponents over [emin, emax]."""
    m = rng.integers(0, 2 ** 52, n, dtype=U)
    return ((rng.integers(0, 2, n, dtype=U) << U(63)) | (rng.integers(emin, emax + 1, n, dtype=U) << U(52)) | m).view(np.float64)


SPECIAL = np.array([0x0000000000000000, 0x8000000000000000, 0x7FF0000000000000, 0xFFF0000000000000, 0x7FF8000000000000,
                    0xFFF8000000000000, 0x7FFFFFFFFFFFFFFF, 0xFFFFFFFFFFFFFFFF, 1, 0x8000000000000001,
                    0x000FFFFFFFFFFFFF, 0x0010000000000000, 0x7FEFFFFFFFFFFFFF, 0xFFEFFFFFFFFFFFFF,
                    0x3FF0000000000000, 0xBFF0000000000000, 0x3FEFFFFFFFFFFFFF, 0x3FF0000000000001], U).view(np.float64)


def _mulhi(a, b):
    m32 = U(0xFFFFFFFF)
    al, ah, bl, bh = a & m32, a >> U(32), b & m32, b >> U(32)
    t = ah * bl + (al * bl >> U(32))
    return ah * bh + (t >> U(32)) + ((al * bh + (t & m32)) >> U(32))


def _hard_quotients(b, r, sign, k):
    """a with a 2^k = b m + sign r for an odd 54-bit m (k = 53: a / b in [1, 2), 54: in [1/2, 1)), where a is a double."""
    inv = b.copy()
    for _ in range(6):
        inv = inv * (U(2) - b * inv)  # b^-1 mod 2^64
    m = (U(0) - inv * r if sign > 0 else inv * r) & U(2 ** k - 1)
    if k == 53:
        m |= U(2 ** 53)
    lo, hi = b * m, _mulhi(b, m)
    a = (hi << U(64 - k)) | (lo >> U(k))
    if sign > 0:
        a += U(1)
    ok = (m >= U(2 ** 53)) & ((a < U(2 ** 53)) | (a & U(1) == 0)) & (a >= U(2 ** 51))
    return a[ok].astype(np.float64), b[ok].astype(np.float64)


def test_quotients(probe):
    rng = np.random.default_rng(1)
    cases = []
    for top in (2.0 ** 53, 2.0 ** 48, 2.0 ** 44, 2.0 ** 40, 2.0 ** 30):  # divisors all over and just below a power of two
        b = (U(2 ** 53) - rng.integers(1, int(min(top, 2 ** 52)), 200_000, dtype=U)) | U(1)
        for r in (1, 3, 5, 9):
            for sign in (1, -1):
                for k in (53, 54):
                    cases.append(_hard_quotients(b, U(r), sign, k))
    a, b = (np.concatenate(c) for c in zip(*cases))
    n = len(a)
    assert n > 5_000_000
    ea, eb = rng.integers(-290, 240, n), rng.integers(-290, 240, n)  # the seeds' range and beyond it
    a, b = np.ldexp(a, ea), np.ldexp(b, eb)
    a *= rng.choice([1.0, -1.0], n)
    R = 2_000_000
    ra = np.concatenate([a, _doubles(rng, R), _doubles(rng, R, 768, 1280), np.repeat(SPECIAL, len(SPECIAL))])
    rb = np.concatenate([b, _doubles(rng, R), _doubles(rng, R, 768, 1280), np.tile(SPECIAL, len(SPECIAL))])
    with np.errstate(all="ignore"):
        want = ra / rb
    _same(probe(3, ra, rb), want, ra, rb)
    near = probe(13, ra, rb)  # physical mode's: an ulp off at most, and only next to a midpoint
    off = np.where(np.isfinite(want), np.abs(_bits(near).astype(np.int64) - _bits(want).astype(np.int64)), 0)
    assert off.max() <= 1 and np.count_nonzero(off[n:n + 2 * R]) == 0  # (none among the random operands)
    np.testing.assert_array_equal(np.isnan(near), np.isnan(want))
    pos = rb > 0  # the vector form divides by a positive length
    for op in (4, 5):
        _same(probe(op, ra[pos], rb[pos]), want[pos], ra[pos], rb[pos])


def test_roots(probe):
    rng = np.random.default_rng(2)
    hard = []
    for K, lo, hi in ((52, 2 ** 52, 6369051672525773), (53, 6369051672525773, 2 ** 53)):  # below and above 2^52.5
        mask = (1 << K) - 1
        for j in range(-20000, 20001, 2):
            for m in (0, 1):
                for _ in range(6):
                    m = (m - (m * m + m + j) * pow(2 * m + 1, -1, 1 << K)) & mask
                for M in (m, m + (1 << 52)):
                    x = M * M + M + j
                    if lo <= M < hi and x & mask == 0:
                        hard.append(x >> K if K == 52 else (x >> K) * 2)
    x = np.array(hard, dtype=U).astype(np.float64)
    assert len(x) > 20_000
    x = np.ldexp(x, 2 * rng.integers(-500, 460, len(x)))
    # the roots whose reciprocal lies closest above a midpoint: divisors of 2^106 - r
    sympy = pytest.importorskip("sympy")
    near = np.array([d for r in range(1, 17) for d in sympy.divisors(2 ** 106 - r) if 2 ** 52 <= d < 2 ** 53],
                    dtype=U).astype(np.float64)
    assert len(near) > 50 and 2.0 ** 53 - 1 in near
    near = np.ldexp(np.tile(near, 8), rng.integers(-250, 200, 8 * len(near)))
    x = np.concatenate([x, near * near, np.abs(_doubles(rng, 4_000_000)), _doubles(rng, 10_000), SPECIAL])
    with np.errstate(all="ignore"):
        s = np.sqrt(x)
        inv = 1.0 / s
    np.testing.assert_array_equal(s[len(x) - len(SPECIAL) - 4_010_000 - len(near):][:len(near)], near)
    _same(probe(0, x), s, x)
    _same(probe(2, x), s, x)
    _same(probe(1, x), inv, x)


def test_conversions(probe):
    rng = np.random.default_rng(3)
    # exponents around the float range, low bits next to a tie
    m = rng.integers(0, 2 ** 52, 3_000_000, dtype=U)
    low = rng.choice(np.array([0, 1, 0x0FFFFFFF, 0x10000000, 0x10000001, 0x1FFFFFFF], U), len(m))
    e = rng.integers(1023 - 155, 1023 + 130, len(m), dtype=U)
    tie = (rng.integers(0, 2, len(m), dtype=U) << U(63)) | (e << U(52)) | (m & ~U(0x1FFFFFFF)) | low
    # ties among the subnormals: a single bit below the last place
    d = rng.integers(0, 53, 500_000, dtype=U)
    sub = (rng.integers(1023 - 151, 1023 - 125, len(d), dtype=U) << U(52)) | ((rng.integers(0, 2 ** 52, len(d), dtype=U) >> d) << d)
    x = np.concatenate([tie.view(np.float64), sub.view(np.float64), _doubles(rng, 2_000_000), SPECIAL])
    with np.errstate(all="ignore"):
        want = x.astype(np.float32)
    got = _bits(probe(6, x)).astype(np.uint32).view(np.float32)
    nan = np.isnan(want)
    assert np.isnan(got[nan]).all()
    np.testing.assert_array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
    u = np.concatenate([rng.integers(0, 2 ** 32, 3_000_000, dtype=np.uint32),
                        rng.integers(0, 2 ** 24, 1_000_000, dtype=np.uint32),  # subnormals and the smallest normals
                        np.arange(2 ** 16, dtype=np.uint32) << np.uint32(16),
                        (np.arange(2 ** 16, dtype=np.uint32) << np.uint32(16)) - np.uint32(1)])
    f = u.view(np.float32)
    with np.errstate(all="ignore"):
        want = f.astype(np.float64)
    _same(probe(7, u.astype(U)), want, f)


def test_comparisons(probe):
    rng = np.random.default_rng(4)
    a = np.concatenate([_doubles(rng, 100_000), SPECIAL])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(probe(9, a) != 0, a <= 0)  # false for a NaN of either sign
        np.testing.assert_array_equal(_bits(probe(10, a)), _bits(np.where(a > 0, a, 0.0)))
        np.testing.assert_array_equal(probe(11, a) != 0, np.isfinite(a))
        _same(probe(12, a), np.where(a == 0, 0.0, a), a)
        # a >= 0 or NaN against b >= 0
        x = rng.permutation(np.abs(a[~np.isnan(a)]))
        y = rng.permutation(x)
        x[:8] = np.tile(SPECIAL[np.isnan(SPECIAL)], 2)
        y[:8] = [0.0, 1.0, np.inf, 1e-8, 1e-300, 5e-324, 1e300, 2.0]
        x[8:2000] = y[8:2000]
        np.testing.assert_array_equal(probe(8, x, y) != 0, x < y)
