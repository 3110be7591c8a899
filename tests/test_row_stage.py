"""Which groups of CSR rows the momentum row kernel stages in shared memory
(nalu-wind_gb300/csrc/row_stage.h, compiled for the host): exactly those that
fit, at any size that the graph limits allow. A size that wraps in 32 bits
must not look small: the kernel would write past its shared memory."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "nalu-wind_gb300" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("row_stage") / "librow_stage.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(so),
                    str(HERE / "row_stage_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


def test_staged_exactly_when_it_fits(lib):
    lib.row_staged.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    sizes = [0, 1, 629, 630, 1535, 1536, 1537, 2047, 2048, 2049]
    sizes += [2 ** k + d for k in range(27, 37) for d in (-1, 0, 1, 630)]
    for smem in (0, 16, 5056, 12288, 16384):
        for first in (0, 1, 2 ** 33 + 1):
            for n in sizes:
                assert bool(lib.row_staged(first, first + n, smem)) == (8 * (n + first % 2) <= smem), (smem, first, n)
