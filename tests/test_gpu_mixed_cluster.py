"""Several steps of a small mesh in one thread-block cluster (mixed path) against the same steps one launch sequence each."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import mesh_of

pytestmark = pytest.mark.gpu

GAM = 2 - 1 / (4 / 3)


@pytest.mark.parametrize("kind,level", [("hex", 0), ("hex", 1), ("hex", 3), ("quad", 2), ("quad", 4), ("ico", 3), ("hex", 4)])
@pytest.mark.parametrize("solver", [1, 2, 3, 4])
def test_steps_together_equal_steps_alone(kind, level, solver, tmp_path):
    """Empty and full blocks, meshes of 3 to 6 edges per face, the largest mesh of one cluster (quad 4: 16 times 192 edges)
    and one beyond, more steps than one launch takes, every solver: the same bits, clock and stop state, whatever runs next."""
    import splash_gb300 as sg

    mesh = mesh_of(kind, level)
    r = sg.Geometry(mesh).unit_face_centers()
    U = sg.initial_conditions.rotating_blob(r, GAM, seed=solver)
    U[:, 0] *= 1 + 1e-2 * np.random.default_rng(level).uniform(-1, 1, len(U))
    dim = 4 if solver == 4 else 5
    U = np.ascontiguousarray(U[:, :dim])
    params = sg.SolverParams(accretion_rate=1e-2, e_acc=0.5, omega_acc_abs=0.5, tilt_angle=0.2, acc_width=0.1,
                             alpha=1e-6, friction_on=solver == 3)
    a, b = (sg.Solver(mesh, U, dim, GAM, 0.0, dim == 5, params=params, solver=solver, precision=sg.PREC_MIXED)
            for _ in range(2))
    for n, dt in ((2, 1e-2), (1, 5e-3), (515, 1e-4), (9, 1.0)):
        a.do_steps(n, dt)
        for _ in range(n):
            b.do_step(dt)
        assert np.array_equal(a.get_state(), b.get_state()), n
        assert a.time() == b.time() and a.last_dt() == b.last_dt() and a.get_stop_check() == b.get_stop_check(), n
    # the writers recompute the last step's edge states
    a.write_t_curl(str(tmp_path / "a.dat"))
    b.write_t_curl(str(tmp_path / "b.dat"))
    assert (tmp_path / "a.dat").read_text() == (tmp_path / "b.dat").read_text()
