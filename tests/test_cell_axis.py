"""The list build's cell of a coordinate (csrc/cell_axis.h, host and device): in
the grid for every float, since the build indexes memory with it, and with the
image in the box as long as a float resolves the box there."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sucrose_gb300", "csrc")


@pytest.fixture(scope="module")
def cell_axis(tmp_path_factory):
    d = tmp_path_factory.mktemp("cell_axis")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text('#include "cell_axis.h"\n'
                   'extern "C" int cell(float* x, int nc, double L) {\n'
                   '    return cell_axis(*x, nc, (float)L, (float)(1.0 / L), L);\n}\n')
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-ffp-contract=off", "-shared", "-fPIC",
                        "-I", CSRC, str(src), "-o", str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(str(lib)).cell
    fn.argtypes = [C.POINTER(C.c_float), C.c_int, C.c_double]

    def call(x, nc, L):
        v = C.c_float(x)
        return fn(C.byref(v), nc, L), v.value
    return call


@pytest.mark.parametrize("L", [3.05, 11.0, 107.3])
def test_cell_is_in_the_grid_for_every_float(cell_axis, L):
    int32 = [-2.0 ** 31, -2.0 ** 31 - 256, 2.0 ** 31, 2.0 ** 31 - 256, -2.0 ** 31 + 128, 2.0 ** 24, -2.0 ** 24]
    for nc in list(range(3, 201)) + [1, 1023, 1024]:
        far = [c * L / nc for c in int32 + [-nc, -1.0, 0.0, nc, 2.0 * nc]]
        for x in far + [np.inf, -np.inf, np.nan, 1e13, -1e13, 1e20, -1e20, 3.4e38, -3.4e38, 0.0, L / 2, -L / 2]:
            assert 0 <= cell_axis(x, nc, L)[0] < nc, (x, nc)


@pytest.mark.parametrize("L", [3.05, 11.0])
def test_image_is_in_the_box_and_in_the_cell(cell_axis, L):
    rng = np.random.default_rng(3)
    for nc in (1, 3, 4, 13, 100):
        for x in np.float32(rng.uniform(-3 * L, 3 * L, 400)):
            c, y = cell_axis(float(x), nc, L)
            boxes = (float(x) - y) / L
            # the image: whole boxes off, to half an ulp; the cell to the FP32 rounding of a few boxes
            assert abs(boxes - round(boxes)) < 1e-6 and abs(y) <= L / 2 * (1 + 2e-6)
            assert c * L / nc - 2e-6 * L <= y + L / 2 <= (c + 1) * L / nc + 2e-6 * L
