"""The limiter in pairs of floats (limiter_pair.cuh) where the ratio nearly vanishes."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_fp64_paths import _p, lib  # noqa: F401


@pytest.mark.parametrize("nu", [4.0, 1e-2, 1e-8, 2.0**-58])
def test_vanishing_ratios_against_the_full_limiter(lib, nu):  # noqa: F811
    """Ratios from 2^-140 to 2^-40 of both signs, with superbee scales up to 2^55: within the 2^-44 of the other ratios, in
    pairs at the Courant factors of a run and wherever pairs are taken."""
    r = np.concatenate([s * np.exp2(np.linspace(-140, -40, 4001)) for s in (1, -1)] + [[0.0, -0.0]])
    dp = np.random.default_rng(3).choice([-1, 1], r.size) * np.exp2(np.linspace(-30, 30, r.size))
    num, nus = r * dp, np.full(r.size, nu)
    pairs, full, served = np.empty_like(r), np.empty_like(r), np.empty(r.size, dtype=np.int32)
    lib.limiter_pairs(len(r), _p(dp), _p(num), _p(nus), ctypes.c_double(1.9), ctypes.c_double(0.16), _p(pairs), _p(full),
                      served.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    assert (served == 1).all() or nu < 1e-6
    assert np.abs(np.where(served == 1, pairs, full) - full).max() <= 2.0**-44
