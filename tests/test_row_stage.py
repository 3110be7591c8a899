"""Which groups of CSR rows the momentum row kernel stages in shared memory
(nalu-wind_gb300/csrc/row_stage.h, compiled for the host): exactly those that
fit, at any size that the graph limits allow. A size that wraps in 32 bits
must not look small: the kernel would write past its shared memory."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
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


@pytest.mark.parametrize("columns", [7, 15, 17, 18, 20, 22])
def test_momentum_rows_of_22_block_columns_are_staged(lib, nw, columns):
    """The staging that the library gives a warp of the momentum row kernel
    (six warps share a block's 96 KB: 16 KB each, 2,048 entries) holds ten
    node rows of up to 22 block columns, whatever their position's parity."""
    f = nw.load()._ZN2nw15row_stage_bytesEiPKll
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_void_p, ctypes.c_int64]
    nodes = 37
    row_ptr = np.arange(3 * nodes + 1, dtype=np.int64) * (3 * columns)
    smem = f(2, row_ptr.ctypes.data, nodes)
    assert smem % 16 == 0 and 6 * smem <= 96 * 1024
    lib.row_staged.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    for first in (0, 1):
        assert lib.row_staged(first, first + 10 * 9 * columns, smem)
