"""Row order of the node-wise Gauss-Seidel sweeps
(nalu-wind_gb300/csrc/gs_order.h, compiled for the host): the classes
(colour, row of the node) in the order of the class-by-class sweep, for the
symmetric sweep and for each half alone."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "nalu-wind_gb300" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("gs_order") / "libgs_order.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(so),
                    str(HERE / "gs_order_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("dof", [2, 3])
@pytest.mark.parametrize("ncol", [1, 2, 3, 8])
@pytest.mark.parametrize("sweep", [0, 1, 2])
def test_node_passes_visit_the_classes_in_sweep_order(lib, dof, ncol, sweep):
    classes, fwd = (ctypes.c_int * (2 * ncol * dof))(), ctypes.c_int()
    n = lib.gs_order(ncol, dof, sweep, classes, ctypes.byref(fwd))
    up = list(range(ncol * dof))
    want = {0: up + up[-2::-1], 1: up, 2: up[::-1]}[sweep]
    assert classes[:n] == want
    assert fwd.value == (0 if sweep == 2 else len(up))
