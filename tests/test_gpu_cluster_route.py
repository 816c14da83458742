"""Which launches do_steps takes on small meshes of the mixed path, and that it takes none while its stream is captured."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import mesh_of

pytestmark = pytest.mark.gpu

GAM = 2 - 1 / (4 / 3)


def _solver(kind, level):
    import splash_gb300 as sg

    mesh = mesh_of(kind, level)
    U = sg.initial_conditions.rotating_blob(sg.Geometry(mesh).unit_face_centers(), GAM, seed=1)
    return sg.Solver(mesh, U, 5, GAM, 0.0, False, params=sg.SolverParams(), solver=3, precision=sg.PREC_MIXED)


@pytest.fixture(scope="module")
def profiler():
    """The profiler's first session in a process starts recording late."""
    from torch.profiler import ProfilerActivity, profile

    s = _solver("hex", 1)
    with profile(activities=[ProfilerActivity.CUDA]):
        s.do_steps(1, 1e-3)
        s.synchronize()
    return lambda: profile(activities=[ProfilerActivity.CUDA])


@pytest.mark.parametrize("kind,level,cluster", [("hex", 0, True), ("hex", 3, True), ("quad", 4, True), ("ico", 3, True),
                                                ("hex", 4, False), ("quad", 5, False)])
def test_meshes_of_up_to_3072_edges_take_the_cluster(profiler, kind, level, cluster):
    """The kernels that ran, by the profiler's record: one cluster launch for eight steps, or 32 launches; one step alone is
    four launches on every mesh."""
    s = _solver(kind, level)
    for n in (8, 1):
        with profiler() as p:
            s.do_steps(n, 1e-3)
            s.synchronize()
        names = [e.name for e in p.events() if "kernel" in e.name and "splash" in e.name]
        if not names:
            pytest.skip("no kernel records from the profiler")
        together = [k for k in names if "cluster_steps_kernel" in k]
        assert len(together) == (1 if cluster and n > 1 else 0), names
        assert len(names) == (1 if together else 4 * n), names


def test_steps_are_refused_during_capture():
    """A solver's steps are graph launches, which a capture refuses; the cluster's are refused alike, leave the capture empty
    and the solver as it was."""
    import splash_gb300 as sg

    cu = C.CDLL("libcuda.so.1")
    a, b = _solver("hex", 3), _solver("hex", 3)
    stream, graph, nodes = C.c_void_p(a.stream()), C.c_void_p(), C.c_size_t(1)
    assert cu.cuStreamBeginCapture_v2(stream, 2) == 0
    with pytest.raises(sg.SplashError):
        a.do_steps(8, 1e-3)
    assert cu.cuStreamEndCapture(stream, C.byref(graph)) == 0
    assert cu.cuGraphGetNodes(graph, None, C.byref(nodes)) == 0 and nodes.value == 0
    cu.cuGraphDestroy(graph)
    for s in (a, b):
        s.do_steps(8, 1e-3)
    assert np.array_equal(a.get_state(), b.get_state()) and a.time() == b.time()
    for s in (a, b):
        n = C.c_int64()
        assert sg.library().splash_steps(s.handle, C.byref(n)) == 0 and n.value == 8
