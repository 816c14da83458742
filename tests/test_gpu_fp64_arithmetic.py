"""The FP64 path's own reciprocal, quotient and root, the switch's table and the limiter in pairs of floats on the device,
where the hardware's seeds (rcp / rsqrt.approx) make them, at the accuracy that fp64_math.cuh and limiter_pair.cuh state."""
from __future__ import annotations

import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = Path(__file__).resolve().parent.parent
PKG = REPO / "muscl-scheme-on-spherical-mesh-wip_gb300"
RECIP, DIVIDE, ROOT, RATIO, SWITCH, LIMITER = range(6)
_D = ctypes.POINTER(ctypes.c_double)
TINY, LEAST, MOST = 5e-324, 2.0**-1022, np.finfo(float).max


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    sys.path.insert(0, str(PKG / "csrc"))
    import importlib.util

    import limiter_table

    spec = importlib.util.spec_from_file_location("splash_build", PKG / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    tmp = tmp_path_factory.mktemp("fp64device")
    limiter_table.write(tmp / "limiter_switch_table.inc")
    out = tmp / "libfp64device.so"
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    *build.CU_FLAGS["step_fp64.cu"], f"-I{tmp}", f"-I{PKG / 'csrc'}", f"-I{REPO / 'include'}",
                    str(REPO / "tests" / "cpp" / "fp64_device.cu"), "-o", str(out)], check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))

    def call(op, *planes, p0=0.0, p1=0.0):
        n = len(planes[0])
        a = np.zeros((3, n))
        for i, p in enumerate(planes):
            a[i] = p
        res = np.empty((3, n))
        assert lib.run(op, n, a.ctypes.data_as(_D), ctypes.c_double(p0), ctypes.c_double(p1), res.ctypes.data_as(_D)) == 0
        return res

    return call


def _same(a, b):
    """Equal bits, any NaN for a NaN."""
    return (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))


def _ulps(a, b):
    """Distance in units of the last place of numbers of equal sign."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def _numbers(rng, n, low=-1074, high=1023):
    """Random mantissas, and those near 1 and 2, over the exponents low .. high; both signs."""
    m = np.concatenate([rng.uniform(1, 2, n), 1 + 2.0**-52 * rng.integers(0, 40, n // 8), 2 - 2.0**-52 * rng.integers(1, 40, n // 8)])
    return rng.choice([-1.0, 1.0], m.size) * np.ldexp(m, rng.integers(low, high + 1, m.size))


EDGES = np.array([s * x for s in (1, -1) for x in (
    0.0, TINY, 3 * TINY, LEAST - TINY, LEAST, 1.5 * LEAST, 2 * LEAST, 4 * LEAST, 8 * LEAST, 1e-305, 1e-300, 1.0, 3.0, 1e300,
    2.0**1020, 2.0**1021, 2.0**1022 - 2.0**969, 2.0**1022 - 2.0**990, 2.0**1022 - 2.0**1000, 2.0**1022 - 2.0**1002,
    2.0**1022, 2.0**1022 + 2.0**970, 1.5 * 2.0**1022, 2.0**1023, MOST, np.inf, np.nan)])


def test_reciprocal(run):
    """1 ulp over the whole range; the operator's bits where it leaves the range of the seeds."""
    rng = np.random.default_rng(1)
    b = np.concatenate([EDGES, _numbers(rng, 2_000_000), _numbers(rng, 200_000, 1018, 1023), _numbers(rng, 200_000, -1024, -1018)])
    with np.errstate(all="ignore"):
        want = 1 / b
    got = run(RECIP, b)[0]
    odd = ~np.isfinite(want) | (np.abs(b) < 2 * LEAST) | (np.abs(b) >= 2.0**1022)
    assert _same(got, want)[odd].all()
    assert (_ulps(got, want) <= 1)[~odd].all(), b[~odd][_ulps(got, want)[~odd] > 1][:5]


def _near_midpoints(rng, n):
    """a, b whose quotient lies as near to the middle of two doubles as quotients come: a 2^54 = b M +- 1 with an odd
    54-bit M, b over all mantissas and near 2."""
    a, b = [], []
    while len(a) < n:
        B = int(rng.integers(2**52, 2**53)) | 1
        if len(a) % 2:
            B = 2**53 - 1 - 2 * int(rng.integers(0, 2**20))
        inv = pow(B, -1, 2**54)
        for s in (1, -1):
            M = (-s * inv) % 2**54
            A = (B * M + s) >> 54
            if M >= 2**53 and (B * M + s) == A << 54 and 2**52 <= A < 2**53:
                a.append(A)
                b.append(B)
    return np.array(a, dtype=float), np.array(b, dtype=float)


def test_quotient_is_the_operators(run):
    """The operator's bits (IEEE division, as numpy's): every pair of edge values, random operands over the whole range,
    numerators whose remainder is subnormal, subnormal quotients, quotients next to the middle of two doubles."""
    rng = np.random.default_rng(2)
    e = np.repeat(EDGES, EDGES.size), np.tile(EDGES, EDGES.size)
    ha, hb = _near_midpoints(rng, 40_000)
    scale = np.ldexp(1.0, rng.integers(-60, 61, ha.size))
    n = 2_000_000
    x, y = _numbers(rng, n), _numbers(rng, n)
    small, one = _numbers(rng, n // 2, -1074, -960), _numbers(rng, n // 2, -40, 40)
    u, w = _numbers(rng, 2 * n, -30, 30), _numbers(rng, 2 * n, -30, 30)
    zero = np.repeat([0.0, -0.0], w.size // 20)
    a = np.concatenate([e[0], ha, ha * scale, x, u, small, one, zero])
    b = np.concatenate([e[1], hb, hb, y, w, one, one * 2.0**980, w[:zero.size]])
    with np.errstate(all="ignore"):
        want = a / b
    got = run(DIVIDE, a, b)[0]
    bad = ~_same(got, want)
    assert not bad.any(), (bad.sum(), a[bad][:5], b[bad][:5], got[bad][:5], want[bad][:5])


def test_slope_ratio(run):
    """2 ulp (a rounded reciprocal and a product), the operator's kind of result where that is no normal number."""
    rng = np.random.default_rng(3)
    e = np.repeat(EDGES, EDGES.size), np.tile(EDGES, EDGES.size)
    a = np.concatenate([e[0], _numbers(rng, 1_000_000, -300, 300)])
    b = np.concatenate([e[1], _numbers(rng, 1_000_000, -300, 300)])
    with np.errstate(all="ignore"):
        want = a / b
    got = run(RATIO, a, b)[0]
    normal = np.isfinite(want) & (np.abs(want) >= 2 * LEAST) & (np.abs(b) < 2.0**1022)
    assert (_ulps(got, want) <= 2)[normal].all()
    assert _same(got, want)[~np.isfinite(want)].all()


def test_root(run):
    """1 ulp, the inverse root 2; the operator's bits for zeros, negative, subnormal, infinite and NaN arguments."""
    rng = np.random.default_rng(4)
    x = np.concatenate([EDGES, np.abs(_numbers(rng, 2_000_000)), rng.uniform(0.5, 4, 1_000_000) ** 2])
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
        iwant = (1 / np.sqrt(x.astype(np.longdouble))).astype(float)
    got, inv, _ = run(ROOT, x)
    odd = ~(x >= 2 * LEAST) | ~(x < 2.0**1022)
    assert _same(got, want)[odd].all()
    assert (_ulps(got, want) <= 1)[~odd].all()
    assert (_ulps(inv, iwant) <= 2)[~odd].all()


def test_switch_table(run):
    """Against the formula in 45-digit arithmetic of the argument that the table takes (below 1 that is 1 - r, rounded), over
    (0, 2.25], near 1 on both sides and at the intervals' ends: 2 ulp of 1 (the row's constant and the sum round once each)."""
    import limiter_table as lt
    from decimal import Decimal

    rng = np.random.default_rng(5)
    d = np.exp2(rng.uniform(-39.9, 0, 1500))
    ends = 1 + np.arange(1, 321) / 256.0
    r = np.concatenate([rng.uniform(0, 2.5, 1500), 1 - d, 1 + d, ends, np.nextafter(ends, 0), [1.0, 1e-300, 1e300]])
    r = r[r > 0]
    got = run(SWITCH, r)[0]
    for x, h in zip(r.tolist(), got.tolist()):
        want = lt.h_below(Decimal(1 - x))[0] if x < 1 else lt.h_above(Decimal(x))[0] if x < 4 else Decimal(1)
        assert abs(float(Decimal(h) - want)) <= 2**-52, x


@pytest.mark.parametrize("eta_p", [1.0, 1.7, 2.24])
def test_limiter_in_pairs_of_floats(run, eta_p):
    """As the host build's test: within 2^-44 of the FP64 limiter, here from the hardware's reciprocal seed."""
    rng = np.random.default_rng(6)
    n = 400_000
    r = np.concatenate([rng.uniform(0, 4, n), 1 + rng.choice([-1, 1], n) * np.exp2(rng.uniform(-52, -1, n)),
                        np.exp(rng.uniform(-30, 30, n)), eta_p * (1 + np.exp2(rng.uniform(-52, -4, n))),
                        1 - np.exp2(-rng.integers(1, 39, n).astype(float)) * (1 + rng.choice([-1e-9, 0, 1e-9], n)),
                        1 + rng.integers(0, 320, n) / 256.0, -rng.uniform(0, 3, n)])
    dp = rng.choice([-1, 1], r.size) * np.exp2(rng.uniform(-200, 200, r.size))
    nu = np.exp(rng.uniform(np.log(1e-5), np.log(4), r.size))
    pairs, full, served = run(LIMITER, dp, r * dp, nu, p0=eta_p, p1=0.16)
    ok = served == 1
    assert ok.mean() > 0.9
    assert np.abs(pairs - full)[ok].max() <= 2.0**-44
