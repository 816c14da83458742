"""Which meshes the FP64 path's edge numbering takes (slot_planes.cpp)."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
CSRC = REPO / "muscl-scheme-on-spherical-mesh-wip_gb300" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("limits") / "liblimits.so"
    sources = [REPO / "tests" / "cpp" / "edge_limits.cpp", CSRC / "slot_planes.cpp", CSRC / "hilbert.cpp", CSRC / "geometry.cpp",
               CSRC / "mesh.cpp"]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-fopenmp", "-Wno-unknown-pragmas", f"-I{CSRC}",
                    f"-I{REPO / 'include'}", *map(str, sources), "-o", str(out)], check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))
    lib.padded.restype = lib.max_adjoint_sides.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("edges,taken", [(1, True), (33, True), (30 * 4**11, True), (12 * 4**12, True), (2**28 - 1, True),
                                         (2**28, True), (2**28 + 1, False), (30 * 4**12, False), (2**31 - 1, False)])
def test_meshes_up_to_quad_12_and_hex_11(lib, edges, taken):
    """What four planes of two sides per edge leave addressable by int, and nothing beyond; the adjoint's codes side * 8 +
    position (up to 4) fit an int over the sides that it takes."""
    pad = lib.padded(edges)
    assert (pad >= 0) == taken
    if taken:
        assert pad % 32 == 0 and edges <= pad < edges + 32 and 4 * 2 * pad - 1 <= 2**31 - 1
    assert (lib.max_adjoint_sides() - 1) * 8 + 4 <= 2**31 - 1
