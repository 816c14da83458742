"""CPU checks of the FP64 path's limiter and fluxes (fp64_math.cuh,
physics_fp64.cuh): the limiter's integer-comparison path gives the general
path's bits, the switch's polynomial table is the switch, and the Riemann
fluxes are the reference's."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
import sys
from decimal import Decimal
from pathlib import Path

import numpy as np
import pytest

from helpers import load, mesh_of

REPO = Path(__file__).resolve().parent.parent
CSRC = REPO / "muscl-scheme-on-spherical-mesh-wip_gb300" / "csrc"
_D = ctypes.POINTER(ctypes.c_double)


def _p(a):
    return a.ctypes.data_as(_D)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    sys.path.insert(0, str(CSRC))
    import limiter_table

    tmp = tmp_path_factory.mktemp("fp64paths")
    limiter_table.write(tmp / "limiter_switch_table.inc")
    out = tmp / "libfp64paths.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    "-DSPLASH_SWITCH_TABLE", f"-I{tmp}", f"-I{CSRC}", f"-I{REPO / 'include'}", str(REPO / "tests" / "cpp" / "fp64_paths.cpp"), "-o", str(out)],
                   check=True, capture_output=True)
    return ctypes.CDLL(str(out))


@pytest.mark.parametrize("eta_p", [0.7, 1.0, 1.9, 2.3])
def test_limiter_positive_path_is_the_general_path(lib, eta_p):
    """Every kind of ratio (zeros, subnormals, infinities, NaN, both signs, the switch's edges) against every positive
    finite superbee scale and a Courant factor from 0 to beyond 2 (a negative third-order line): the same bits."""
    rng = np.random.default_rng(1)
    edge = [0.0, 5e-324, 1e-300, 2.0**-16, 1 - 2.0**-16, 1 - 2.0**-17, 1 - 2.0**-53, 1.0, 1 + 2.0**-52, 2.0, 2.25,
            2.25 - 2.0**-51, 3.0, 1e300, np.inf, np.nan, eta_p, np.nextafter(eta_p, 3)]
    r = np.concatenate([edge, -np.array(edge), rng.uniform(-3, 5, 4000), np.exp(rng.uniform(-40, 40, 2000))])
    sb = np.exp(rng.uniform(-12, 12, r.size))
    sb[::97] = 1e-310
    nu = np.where(rng.random(r.size) < 0.8, rng.uniform(0, 0.2, r.size), rng.uniform(0, 6, r.size))
    a, b = np.empty_like(r), np.empty_like(r)
    lib.limiter_both(len(r), _p(r), _p(sb), _p(nu), ctypes.c_double(eta_p), _p(a), _p(b))
    assert np.array_equal(a, b)
    assert (a > 0).any() and np.isfinite(a).all()


@pytest.mark.parametrize("eta_p", [1.0, 1.7, 2.24])
def test_limiter_in_pairs_of_floats(lib, eta_p):
    """Against the FP64 limiter, with ratios over the whole range, near 1, near the switch's table edges and near eta_p,
    differences of every size and sign, Courant factors from 1e-5 to 4: within 2^-44 (the ratio and its distance from 1
    carry 2^-46 each; they reach the value with weights up to 2.3 and with the switch's slope, up to 5.6 there where the
    distance is below 1)."""
    rng = np.random.default_rng(2)
    n = 400_000
    r = np.concatenate([rng.uniform(0, 4, n), 1 + rng.choice([-1, 1], n) * np.exp2(rng.uniform(-52, -1, n)),
                        np.exp(rng.uniform(-30, 30, n)), eta_p * (1 + np.exp2(rng.uniform(-52, -4, n))),
                        1 - np.exp2(-rng.integers(1, 39, n).astype(float)) * (1 + rng.choice([-1e-9, 0, 1e-9], n)),
                        1 + rng.integers(0, 320, n) / 256.0, -rng.uniform(0, 3, n)])
    dp = rng.choice([-1, 1], r.size) * np.exp2(rng.uniform(-200, 200, r.size))
    num = r * dp
    nu = np.exp(rng.uniform(np.log(1e-5), np.log(4), r.size))
    pairs, full, served = np.empty_like(r), np.empty_like(r), np.empty(r.size, dtype=np.int32)
    lib.limiter_pairs(len(r), _p(dp), _p(num), _p(nu), ctypes.c_double(eta_p), ctypes.c_double(0.16), _p(pairs), _p(full),
                      served.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    ok = served == 1
    assert ok.mean() > 0.9
    assert np.abs(pairs - full)[ok].max() <= 2.0**-44


def test_limiter_pairs_leave_the_odd_cases(lib):
    """Zero, subnormal, infinite and NaN differences, ratios past 2^60 or within 2^-40 below 1, and Courant factors that
    are not positive and finite are left to FP64; a vanishing numerator gives 0."""
    tiny, inf, nan = 5e-324, np.inf, np.nan
    dp = np.array([0.0, tiny, inf, nan, 1.0, 1.0, 1.0, 1e-300, 1.0, 1.0, 1.0, 1.0, 1.0, 3.0, 1.0])
    num = np.array([1.0, 1.0, 1.0, 1.0, inf, nan, 1 - 2.0**-45, 1.0, 0.5, 0.5, 0.5, 0.5, 0.5, 0.0, -0.5])
    nu = np.array([0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.0, -0.1, inf, nan, 1e-30, 0.1, 0.1])
    pairs, full, served = np.empty_like(dp), np.empty_like(dp), np.empty(dp.size, dtype=np.int32)
    lib.limiter_pairs(len(dp), _p(dp), _p(num), _p(nu), ctypes.c_double(2.0), ctypes.c_double(0.16), _p(pairs), _p(full),
                      served.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    assert list(served) == [0] * 13 + [1, 1]
    assert pairs[-2] == pairs[-1] == 0.0


def test_switch_table_is_the_switch():
    """Each row at its two ends and inside, its polynomial evaluated in double as the kernels do (without their fused
    rounding): h within 2 ulp of 1 (the row's constant and the sum round once each), dh/dr within 1e-14 of the larger
    of 1 and itself (its coefficients are up to 64 times its value per half width)."""
    sys.path.insert(0, str(CSRC))
    import limiter_table as lt

    value, slope = lt.tables()
    assert len(value) == len(slope) == lt.ROWS == 1568
    for i, (centre, half, formula) in enumerate(lt.rows()):
        for x in (-1.0, -0.37, 0.0, 0.61, 1.0):
            d = float(half) * x
            h, g = formula(centre + Decimal(d))
            assert abs(float(Decimal(_horner(value[i], d)) - h)) <= 2**-52, (i, x)
            assert abs(float(Decimal(_horner(slope[i], d)) - g)) <= 1e-14 * max(1.0, abs(float(g))), (i, x)


def _horner(row, d):
    a = 0.0
    for c in reversed(row):
        a = a * d + c
    return a


@pytest.mark.parametrize("case", ["hllep", "hllc", "hllcp"])
def test_fluxes_known_answers(lib, case):
    """Against the reference's own flux_star on its 300 states: within 1e-12 of the flux's scale (the fastest signal
    times the largest state and pressure; some 100 roundings of 1.1e-16 each)."""
    import splash_gb300 as sg

    f = load(f"funcs_{case}.npz")
    g = sg.Geometry(mesh_of(str(f["mesh"]), int(f["level"])))
    gam, off = float(f["gam"]), g["face_off"]
    F = np.empty(5)
    for i in range(len(f["face"])):
        s = off[f["face"][i]] + int(f["edge"][i])
        nxt = s + 1 if s + 1 < off[f["face"][i] + 1] else off[f["face"][i]]
        ec = g["vertices"][g["face_vtx"][s]] + g["vertices"][g["face_vtx"][nxt]]
        ec = np.ascontiguousarray(ec / np.linalg.norm(ec))
        en = np.ascontiguousarray(g["edge_normals"][s])
        uL, uR = np.ascontiguousarray(f["ul"][i]), np.ascontiguousarray(f["ur"][i])
        lib.flux(_p(uL), _p(uR), _p(ec), _p(en), ctypes.c_double(gam), int(f["solver"]), _p(F))
        speed = max(np.linalg.norm(u[1:4]) / u[0] + np.sqrt(gam * gam * abs(u[4]) / u[0]) for u in (uL, uR))
        scale = (1 + speed) ** 2 * max(np.abs(uL).max(), np.abs(uR).max())
        assert np.all(np.abs(F - f["F"][i]) <= 1e-12 * scale), (i, F, f["F"][i])
