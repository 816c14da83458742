"""The extra dt constraint 0.01 Sigma / (alpha rho |v - v0|) and its sign (physics/adiabatic.hpp:543-580) in the FP64 path's
fold: the smallest candidate bounds dt, a negative one stops the run and leaves 1e20."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import make_oracle, mesh_of, rel_linf

REPO = Path(__file__).resolve().parent.parent
CSRC = REPO / "muscl-scheme-on-spherical-mesh-wip_gb300" / "csrc"
GAM = 2 - 1 / (4 / 3)
ALPHAS = [1e-6, 30.0, 0.0, -0.0, -1e-6, -30.0]
_D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def bounds(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("dtbounds") / "libdtbounds.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    f"-I{CSRC}", f"-I{REPO / 'include'}", str(REPO / "tests" / "cpp" / "dt_bounds.cpp"), "-o", str(out)],
                   check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))

    def call(w, r, omega_ns, alpha, h0):
        res = np.empty(4)
        w, r = np.ascontiguousarray(w), np.ascontiguousarray(r)
        d = ctypes.c_double
        lib.dt_bounds_of(len(w), w.ctypes.data_as(_D), r.ctypes.data_as(_D), d(GAM), d(omega_ns), d(alpha), d(h0),
                         res.ctypes.data_as(_D))
        return res

    return call


def _faces(rng, n, speed):
    r = rng.standard_normal((n, 3))
    r /= np.linalg.norm(r, axis=1, keepdims=True)
    v = np.cross(r, rng.standard_normal((n, 3)))
    v *= speed / np.linalg.norm(v, axis=1, keepdims=True)
    sigma, pi = np.exp(rng.uniform(-2, 2, n)), np.exp(rng.uniform(-3, 1, n))
    return r, v, np.column_stack([sigma, sigma[:, None] * np.cross(r, v), pi])


@pytest.mark.parametrize("alpha", ALPHAS + [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("speed", ["slow", "fast", "both"])
def test_bounds_are_the_formulas(bounds, alpha, speed):
    """g_eff = 0.217909 - |v|^2 above 0, below, and of both signs among the faces, every sign and the odd values of alpha:
    the flag exactly, max_vel and the extra dt to 1e-13 (some 20 roundings of 1.1e-16, twice where the fold squares)."""
    rng = np.random.default_rng(4)
    low, high = {"slow": (0.05, 0.4), "fast": (0.6, 1.2), "both": (0.05, 1.2)}[speed]
    r, v, w = _faces(rng, 200, rng.uniform(low, high, (200, 1)))
    omega, h0 = 0.2, 1e-2
    g3 = 1 / (2 - GAM)
    rel = np.linalg.norm(v - np.cross([0, 0, omega], r), axis=1)
    with np.errstate(all="ignore"):
        rho = g3 / (2 * g3 - 1) * (0.217909 - (v * v).sum(1)) * w[:, 0] ** 2 / w[:, 4]
        cand = 0.01 * w[:, 0] / (alpha * rho * rel)
    extra = min([1e20] + [float(c) for c in cand if c < 1e20])
    negative = extra < 0
    if negative:
        extra = 1e20
    vmax = max(np.sqrt((v * v).sum(1)).max(), np.sqrt(GAM * w[:, 4] / w[:, 0]).max())
    got = bounds(w, r, omega, alpha, h0)
    assert bool(got[3]) == negative
    np.testing.assert_allclose(got[:3], [vmax, extra, min(h0 * 0.1 / vmax, extra)], rtol=1e-13, atol=0)



@pytest.mark.gpu
@pytest.mark.parametrize("alpha", ALPHAS)
@pytest.mark.parametrize("speed", ["slow", "fast", "both"])
def test_step_takes_the_oracles_dt_and_stop(alpha, speed):
    """Below sqrt(GM) everywhere, above it everywhere, and both: one step in every way that takes it, FP64 (step, the
    adjoint's forward, the tangent model) and mixed, has the oracle's dt and stop bit, and its state within the parity tests'
    1e-10 (mixed: 1e-6, a few FP32 roundings)."""
    import splash_gb300 as sg
    from splash_gb300.initial_conditions import rotating_blob, to_conserved

    mesh = mesh_of("hex", 3)
    g = sg.Geometry(mesh)
    r = g.unit_face_centers()
    if speed == "fast":
        phi = np.cross([0.36, 0.48, 0.8], r)  # about an axis that is no face centre
        U = to_conserved(r, np.ones(len(r)), np.ones(len(r)), 0.8 * phi / np.linalg.norm(phi, axis=1, keepdims=True), GAM)
    else:
        U = rotating_blob(r, GAM, omega=0.3 if speed == "slow" else 0.9, seed=2)
    params = sg.SolverParams(accretion_rate=1e-2, e_acc=0.5, omega_acc_abs=0.5, tilt_angle=0.2, acc_width=0.1, alpha=alpha,
                             friction_on=True)
    o = make_oracle(g, dict(U0=U, gam=GAM, accretion_on=True, params=params.as_list(), solver=3))
    bits = o.do_step(1.0)
    dt, want = o.info()["dt"], o.get_state()
    assert dt > 0 and bool(bits & sg.STOP_NEG_EXTRA_DT) == (speed == "both" or (speed == "fast") != (np.signbit(alpha)))
    for precision, tol in ((sg.PREC_FP64, 1e-10), (sg.PREC_MIXED, 1e-6)):
        s = sg.Solver(mesh, U, 5, GAM, 0.0, True, params=params, solver=3, precision=precision)
        s.do_step(1.0)
        assert s.error_word() == bits, (precision, s.error_word(), bits)
        assert abs(s.last_dt() - dt) <= tol * dt
        assert np.all(rel_linf(s.get_state(), want) < tol)
        if precision == sg.PREC_FP64:
            adj, theta = sg.Adjoint(s, checkpoint_every=1), np.array([1e-2, 0.2, 0.5])
            assert np.array_equal(adj.forward(U, theta, 1, 1.0), s.get_state())
            assert adj.dt_schedule()[0] == s.last_dt() and adj.error_word() == bits
            assert np.array_equal(adj.tlm(U, theta, np.ones_like(U), np.zeros(3), 1, 1.0)[0], s.get_state())
