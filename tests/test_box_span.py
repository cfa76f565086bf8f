"""box_span (puncpp_gb300/csrc/mesh_tables.cpp): which meshes are boxes without
an inner wall, where a walk may start again near its point, and how many cells
lie between any cell of them and the first one."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import box_meshes
from puncpp_gb300 import meshgen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "puncpp_gb300", "csrc")


@pytest.fixture(scope="module")
def span(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("span") / "libspan.so"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I" + CSRC,
                        "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "box_span.cpp"),
                        os.path.join(CSRC, "mesh_tables.cpp"), "-o", str(so), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(str(so)).box_span_of
    fn.restype = C.c_int64
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int64]

    def call(ma):
        return fn(ma.coords.ctypes.data, ma.n_vertices, ma.cells.ctypes.data, ma.n_cells, ma.bfacets.ctypes.data,
                  ma.btags.ctypes.data, len(ma.btags))

    return call


def test_boxes_with_walls_are_no_boxes(span):
    assert span(box_meshes.plate()) == 0
    assert span(box_meshes.speck()[0]) == 0
    assert span(box_meshes.side_by_side()[0]) == 0
    assert span(meshgen.probe_box(9, 2.0, 0.7)) == 0
    assert span(meshgen.sphere_shell(1.0, 4.0, 1)) == 0


@pytest.mark.parametrize("n", [1, 2, 5, 11])
def test_span_of_a_box(span, n):
    """The cells lie between planes x, y, z = k h and x-y, x-z, y-z = k h, and a
    walk from one to another crosses each plane between them once: counted for
    the first cell at each corner."""
    ma = meshgen.kuhn_box(n, -1.0, 1.0)
    p = (ma.coords[ma.cells] + 1.0) * n / 2
    first = {}
    for k, v in zip(*np.nonzero(np.all((p == 0) | (p == n), axis=2))):
        first.setdefault(tuple(p[k, v]), k)
    c = p[sorted(first.values())].mean(axis=1)
    f = np.floor(np.stack([c[:, 0], c[:, 1], c[:, 2], c[:, 0] - c[:, 1], c[:, 0] - c[:, 2], c[:, 1] - c[:, 2]]))
    assert len(first) == 8
    assert span(ma) == max(1, np.abs(f[:, :, None] - f[:, None, :]).sum(axis=0).max())


def test_span_of_a_slender_box(span):
    assert 3 * 300 - 3 <= span(box_meshes.slender(300)) <= 3 * 300 + 3
