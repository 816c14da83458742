"""The FP64 path on given meshes whose edges it cannot pair (slot_planes.cpp: one edge per slot)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_oracle, mesh_of, rel_linf

GAM = 2 - 1 / (4 / 3)
MESHES = [("quad", 4, 12.0), ("hex", 3, 14.0), ("hex", 4, 8.0), ("hex", 5, 4.0)]


def clockwise_mesh(kind, level, factor):
    """A generated mesh with its faces' corners in clockwise order, drawn together towards the pole by `factor`.  An edge's
    normal is turned outward only where that shows at a distance of 0.01 (MUSCL_geometry.hpp: the normal's sign test), so
    where the faces shrink past that size the normals of an edge's two sides point the same way."""
    import splash_gb300 as sg

    g = sg.Geometry(mesh_of(kind, level))
    x, off, vtx = np.asarray(g["vertices"]).reshape(-1, 3), g["face_off"], g["face_vtx"]
    p = x[:, :2] / np.maximum(1 + x[:, 2:], 1e-9) / factor  # stereographic, from the south pole
    q = (p * p).sum(1, keepdims=True)
    new = np.concatenate([2 * p, 1 - q], axis=1) / (1 + q)
    new[x[:, 2] < -1 + 1e-12] = [0, 0, -1]
    return sg.Mesh(vertices=new, face_offsets=off, face_vertices=np.concatenate([vtx[a:b][::-1] for a, b in zip(off, off[1:])]))


def _geometry(mesh):
    """The mesh's geometry and which slots' normals are not the opposite of their reverse slots'."""
    import splash_gb300 as sg

    g = sg.Geometry(mesh)
    off, nbr, en = g["face_off"], g["nbr_edge"], np.asarray(g["edge_normals"]).reshape(-1, 3)
    face = np.repeat(np.arange(g.n_faces), np.diff(off))
    slot = {(int(f), int(b)): s for s, (f, b) in enumerate(zip(face, nbr))}
    rev = np.array([slot[int(b), int(f)] for f, b in zip(face, nbr)])
    return g, (en != -en[rev]).any(1)


@pytest.mark.parametrize("kind,level,factor", MESHES)
def test_meshes_have_both_kinds_of_edges(kind, level, factor):
    """What the test below is about: some edges are paired, some are not."""
    odd = _geometry(clockwise_mesh(kind, level, factor))[1]
    assert 4 < odd.sum() < len(odd) - 4


@pytest.mark.gpu
@pytest.mark.parametrize("kind,level,factor", MESHES)
@pytest.mark.parametrize("solver", [1, 2, 3, 4])
def test_unpaired_edges_against_the_oracle(kind, level, factor, solver):
    """Few and many edges (a thread per field of a side, and per side): three steps within the parity tests' 1e-10 of the
    oracle, whose faces each evaluate their own edges; the tangent model's values and the recorded forward's are the step's,
    and the gradient is the tangent's transpose to 1e-9 (the rounding of two long sums)."""
    import splash_gb300 as sg

    mesh = clockwise_mesh(kind, level, factor)
    g, _ = _geometry(mesh)
    U = sg.initial_conditions.rotating_blob(g.unit_face_centers(), GAM, seed=solver)
    U[:, 0] *= 1 + 1e-2 * np.random.default_rng(1).uniform(-1, 1, len(U))
    U = np.ascontiguousarray(U[:, :4] if solver == 4 else U)
    dim = U.shape[1]
    params = sg.SolverParams(accretion_rate=1e-2, e_acc=0.5, omega_acc_abs=0.5, tilt_angle=0.2, acc_width=0.1, alpha=1e-6,
                             friction_on=True)
    o = make_oracle(g, dict(U0=U, gam=GAM, accretion_on=dim == 5, params=params.as_list(), solver=solver), dim=dim)
    o.do_steps(3, 1e-5)
    want = o.get_state()
    assert np.isfinite(want).all()
    s = sg.Solver(mesh, U, dim, GAM, 0.0, dim == 5, params=params, solver=solver, precision=sg.PREC_FP64)
    s.do_steps(3, 1e-5)
    got = s.get_state()
    assert np.all(rel_linf(got, want) < 1e-10), rel_linf(got, want)
    if dim == 4:
        return
    adj, theta = sg.Adjoint(s, checkpoint_every=2), np.array([1e-2, 0.2, 0.5])
    rng = np.random.default_rng(2)
    dU, lam = rng.standard_normal(U.shape) * np.abs(U).max(0), rng.standard_normal(U.shape)
    Ut, dUt = adj.tlm(U, theta, dU, np.zeros(3), 3, 1e-5)
    assert np.array_equal(Ut, got) and np.array_equal(adj.forward(U, theta, 3, 1e-5), got)
    grad, _ = adj.backward(lam)
    a, b = (lam * dUt).sum(), (grad * dU).sum()
    assert abs(a - b) <= 1e-9 * np.abs(lam * dUt).sum(), (a, b)
    assert np.array_equal(adj.branch_tape(U, theta, 3, "record")[0], got)
