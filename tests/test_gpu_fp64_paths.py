"""The FP64 step's launches on meshes on either side of its dispatch."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import mesh_of

pytestmark = pytest.mark.gpu

GAM = 2 - 1 / (4 / 3)


@pytest.mark.parametrize("kind,level", [("hex", 2), ("hex", 3), ("hex", 5), ("quad", 5), ("quad", 6), ("quad", 7), ("hex", 7)])
@pytest.mark.parametrize("solver,friction", [(1, True), (2, False), (3, True)])
def test_step_equals_the_tangent_models_values(kind, level, solver, friction):
    """Small meshes update with six threads per face, large ones with one, the tangent-linear model always with six and on
    dual numbers: the same bits, with full and partial last blocks, shallow and steep differences, a clipped dt."""
    import splash_gb300 as sg

    mesh = mesh_of(kind, level)
    r = sg.Geometry(mesh).unit_face_centers()
    U = sg.initial_conditions.rotating_blob(r, GAM, seed=solver)
    U[:, 0] *= 1 + 1e-3 * np.random.default_rng(level).uniform(-1, 1, len(U))
    params = sg.SolverParams(accretion_rate=1e-2, e_acc=0.5, omega_acc_abs=0.5, tilt_angle=0.2, acc_width=0.1,
                             alpha=1e-6, friction_on=friction)
    base = sg.Solver(mesh, U, 5, GAM, 0.0, True, params=params, solver=solver, precision=sg.PREC_FP64)
    adj = sg.Adjoint(base, checkpoint_every=1)
    theta = np.array([1e-2, 0.2, 0.5])
    Ut, _ = adj.tlm(U, theta, np.ones_like(U), np.zeros(3), 3, 1e-2)
    base.do_steps(3, 1e-2)
    assert np.array_equal(base.get_state(), Ut)
    assert base.last_dt() < 1e-2 or level < 4


@pytest.mark.parametrize("kind,level", [("hex", 0), ("hex", 1), ("quad", 1), ("ico", 2), ("hex", 4), ("quad", 5)])
@pytest.mark.parametrize("solver,noise", [(1, 0.2), (2, 1e-3), (3, 1e-2)])
def test_fields_on_threads_of_their_own(kind, level, solver, noise):
    """The smallest meshes give every field of a side a thread, in the step and on dual numbers in the tangent model: the
    same values, with partial blocks (30, 120, 24, 480 edges), up to the largest such mesh, smooth and steep, and the
    recorded forward's, which one thread per face makes."""
    import splash_gb300 as sg

    mesh = mesh_of(kind, level)
    r = sg.Geometry(mesh).unit_face_centers()
    U = sg.initial_conditions.rotating_blob(r, GAM, seed=solver)
    U[:, 0] *= 1 + noise * np.random.default_rng(level).uniform(-1, 1, len(U))
    params = sg.SolverParams(accretion_rate=1e-2, e_acc=0.5, omega_acc_abs=0.5, tilt_angle=0.2, acc_width=0.1,
                             alpha=1e-6, friction_on=True)
    base = sg.Solver(mesh, U, 5, GAM, 0.0, True, params=params, solver=solver, precision=sg.PREC_FP64)
    adj, theta = sg.Adjoint(base, checkpoint_every=1), np.array([1e-2, 0.2, 0.5])
    Ut, _ = adj.tlm(U, theta, np.ones_like(U), np.zeros(3), 5, 1e-3)
    base.do_steps(5, 1e-3)
    # equal_nan: the coarsest quad mesh leaves the range of the method, on both paths alike
    assert np.array_equal(base.get_state(), Ut, equal_nan=True)
    assert np.array_equal(adj.forward(U, theta, 5, 1e-3), Ut, equal_nan=True)
    assert np.array_equal(adj.branch_tape(U, theta, 5, "record")[0], Ut, equal_nan=True)
