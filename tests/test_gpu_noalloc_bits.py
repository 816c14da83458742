"""splash_cfl_dt_noalloc gives the FP64 solver's dt bit for bit, as its declaration says, whichever bound is the smallest."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import mesh_of

pytestmark = pytest.mark.gpu

GAM = 2 - 1 / (4 / 3)


@pytest.mark.parametrize("kind,level", [("hex", 1), ("hex", 4), ("quad", 6)])
@pytest.mark.parametrize("omega,alpha", [(0.2, 1e-6), (3.0, 1e-6), (0.2, 30.0), (0.2, 3e4), (0.9, -30.0), (0.0, 0.0)])
def test_dt_is_the_solvers(kind, level, omega, alpha):
    """The sound speed, the flow speed, the extra constraint, its stop and no extra constraint at all decide; ten states each,
    the solver's clip of dt0 = 1 against the call's, and its flag against the stop bit."""
    torch = pytest.importorskip("torch")
    import splash_gb300 as sg

    lib = sg.library()
    p, d = C.c_void_p, C.c_double
    lib.splash_cfl_dt_noalloc.argtypes = [p, p, p, C.c_int, d, d, d, d, d, p, p]
    mesh = mesh_of(kind, level)
    g = sg.Geometry(mesh)
    r = g.unit_face_centers()
    dr, da = torch.from_numpy(np.ascontiguousarray(r)).cuda(), torch.from_numpy(np.ascontiguousarray(g["area"])).cuda()
    out = torch.empty(9, dtype=torch.float64, device="cuda")
    for seed in range(10):
        U = sg.initial_conditions.rotating_blob(r, GAM, seed=seed, omega=omega)
        s = sg.Solver(mesh, U, 5, GAM, 0.1, False, params=sg.SolverParams(alpha=alpha), solver=2, precision=sg.PREC_FP64)
        s.do_step(1.0)
        dU = torch.from_numpy(U).cuda()
        torch.cuda.synchronize()
        rc = lib.splash_cfl_dt_noalloc(dU.data_ptr(), dr.data_ptr(), da.data_ptr(), len(U), GAM, 0.1, alpha, g.h0, 1.0,
                                       out.data_ptr(), None)
        assert rc == 0
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert got[0] == s.last_dt(), (seed, got[0], s.last_dt())
        assert bool(got[3]) == bool(s.error_word() & sg.STOP_NEG_EXTRA_DT)
        s.close()
