"""Device code that whole steps reach only by luck, called directly through
tests/device_checks.cu: the branch-free divisions (hg_phys.cuh) against the
host's own division at the ends of their ranges, and the FP32 flux kernels
without a geometry's known zeros (hg_mixed.cu) against the ones that take every
entry, on states with infinities."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import coolharm3d_b200 as hg
import fixtures
from coolharm3d_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("checks") / "device_checks.so")
    ctypes.CDLL(hg.LIB_PATH, mode=ctypes.RTLD_GLOBAL)  # hg::launch_flux_f32
    subprocess.check_call([build.nvcc()] + build.flags() + ["-shared", "-o", out, os.path.join(HERE, "device_checks.cu")])
    return ctypes.CDLL(out)


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def operands(rng, n):
    """Numerators and denominators: mantissas at random, of 53 ones, with a low
    word of 32 ones and of a single bit; exponents over both ranges, at their
    ends and beyond; zeros, subnormals, infinities and NaN among them."""
    def numbers(span, edge):
        m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
        kind = rng.integers(0, 8, n)
        m[kind == 0] = (1 << 52) - 1
        m[kind == 1] |= (1 << 32) - 1
        m[kind == 2] = 0
        m[kind == 3] = 1
        e = rng.integers(-span, span + 1, n)
        at = rng.random(n) < 0.2
        e[at] = rng.choice([-edge - 1, -edge, -edge + 1, edge - 1, edge, edge + 1], at.sum())
        e[rng.random(n) < 0.3] = 0
        x = np.ldexp((m | np.uint64(1023 << 52)).view(np.float64), e) * rng.choice([-1.0, 1.0], n)
        special = [0.0, -0.0, 5e-324, 2.0 ** -1022, 1.7e308, np.inf, -np.inf, np.nan]
        odd = rng.random(n) < 0.02
        x[odd] = rng.choice(special, odd.sum())
        return x
    return numbers(1000, 500), numbers(800, 400)


def in_range(x, e):
    return (np.abs(x) >= 2.0 ** -e) & (np.abs(x) < 2.0 ** e)


def test_fast_divisions_round_as_the_host_divides(checks):
    n = 1 << 20
    a, b = operands(np.random.default_rng(1), n)
    out, ok = np.empty((5, n)), np.empty((5, n), np.uint8)
    assert checks.check_divisions(n, ptr(a), ptr(b), ctypes.c_double(1e-10), ptr(out), ptr(ok)) == 0
    ok = ok.astype(bool)
    with np.errstate(all="ignore"):
        quo, rec = a / b, 1.0 / b
    ones = (b.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)
    low = (b.view(np.uint64) & np.uint64(0xffffffff)) == np.uint64(0xffffffff)
    num, den, zero = in_range(a, 500), in_range(b, 400), a == 0
    # exactly the operands of the stated ranges are taken
    assert np.array_equal(ok[0], (num | zero) & den & ~low)
    assert np.array_equal(ok[1], den & ~low)
    assert np.array_equal(ok[2], den)
    assert np.array_equal(ok[3], (num | zero) & den)
    pos = ~(ones & (b < 0))  # rcp_any and div_any: b of 53 ones is positive
    for q, want, take in ((0, quo, ok[0]), (1, rec, ok[1]), (2, rec, ok[2] & pos), (3, quo, ok[3] & pos & ~zero)):
        assert take.sum() > n // 10 and (q < 2 or (take & ones).sum() > 1000)
        assert np.array_equal(out[q][take].view(np.uint64), want[take].view(np.uint64)), q


@pytest.mark.parametrize("tol", [1e-10, 0.3])
def test_within_decides_as_the_rounded_quotient(checks, tol):
    n = 1 << 18
    rng = np.random.default_rng(2)
    x = np.ldexp(1 + rng.random(n), rng.integers(-300, 300, n)) * rng.choice([-1.0, 1.0], n)
    d = np.abs(x) * tol * (1 + rng.integers(-12, 13, n) * 2.0 ** -52) * rng.choice([-1.0, 1.0], n)
    far = rng.random(n) < 0.3
    d[far] *= 10.0 ** rng.uniform(-3, 3, far.sum())
    for v in (0.0, np.inf, np.nan):
        d[rng.integers(0, n, 50)] = v
        x[rng.integers(0, n, 50)] = v
    out, ok = np.empty((5, n)), np.empty((5, n), np.uint8)
    assert checks.check_divisions(n, ptr(d), ptr(x), ctypes.c_double(tol), ptr(out), ptr(ok)) == 0
    with np.errstate(all="ignore"):
        want = np.abs(d / x) <= tol
    ok = ok[4].astype(bool)
    assert ok.sum() > n // 2 and (~ok).sum() > 0
    assert np.array_equal(out[4][ok] != 0, want[ok])


def wild(p, seed):
    """The states in FP32 with some velocities and fields zero, and infinite
    components in a tenth of the zones."""
    rng = np.random.default_rng(seed)
    p = np.ascontiguousarray(p, np.float32)
    p[2:][rng.random(p[2:].shape) < 0.15] = 0
    z = rng.random(p.shape) < 0.02
    p[z] = rng.choice(np.array([np.inf, -np.inf], np.float32), z.sum())
    return p


def classes(x):
    return np.where(np.isnan(x), 2, np.where(np.isposinf(x), 3, np.where(np.isneginf(x), 4, 0)))


@pytest.mark.parametrize("flux", [0, 1])
@pytest.mark.parametrize("strip_nf,strip_x1", [(1, 1), (2, 1), (3, 1), (3, 0)])
@pytest.mark.parametrize("kind", ["flat", "table"])
def test_fp32_known_zeros_keep_infinities(checks, kind, strip_nf, strip_x1, flux):
    rng = np.random.default_rng(6)
    if kind == "flat":
        n, mdim, gk, gam = (10, 7, 6), 0, 1, 4 / 3
        geom = np.zeros(42)
        geom[[0, 16]] = -1
        geom[[5, 10, 15, 21, 26, 31, 32, 33, 34, 38]] = 1
        p0 = rng.uniform(-1, 1, (8,) + tuple(x + 6 for x in n)[::-1])
        p0[:2] += 1.1
    else:
        f = fixtures.load("torus_24x16x8_s1")
        n, mdim, gk, gam = f["n"], 2, 2, f["gam"]
        # rows in the tables' order, x1 fastest
        geom = np.ascontiguousarray(np.array(f["geom"], float).reshape(5, n[0] + 6, n[1] + 6, 42).transpose(0, 2, 1, 3))
        p0 = np.array(f["p0"]).transpose(3, 2, 1, 0)
        p0 = p0 * (1 + 0.1 * rng.uniform(-1, 1, p0.shape))
    shape = p0.shape[1:]
    p = wild(p0, 7)
    nn = np.array(n, np.int32)
    out = []
    for known in (gk, 0):
        F, maxs, booked = np.empty((3, 8) + shape), np.empty(3), np.empty(shape, np.uint32)
        rc = checks.check_flux_f32(ptr(nn), 2, flux, mdim, known, strip_nf, strip_x1, ctypes.c_double(gam), ptr(p), ptr(geom),
                                   ptr(F), ptr(maxs), ptr(booked))
        assert rc == 0
        out.append((F, maxs, booked))
    a, b = out
    assert np.isinf(b[0]).any() and np.isnan(b[0]).any() and np.isfinite(b[0]).any()
    assert np.array_equal(classes(a[0]), classes(b[0]))
    assert np.array_equal(a[2], b[2])
    # finite faces: some 60 FP32 roundings, which the root of a discriminant
    # that cancels turns into their square root
    tol = np.sqrt(60 * 2.0 ** -24)
    fin = np.isfinite(b[0])
    for d in range(3):
        scale = np.abs(b[0][d][fin[d]]).max()
        assert np.abs(a[0][d][fin[d]] - b[0][d][fin[d]]).max() < tol * scale
    assert np.allclose(a[1], b[1], rtol=tol, atol=0)
