"""Error of the float-pair reciprocal that starts from an approximate seed
(dd_rcp_seed in nalu-wind_gb300/csrc/dd.h, compiled for the host) against
extended precision, for every seed within 2^-21 of 1 / x, so also for the
approximate instruction's (one unit in the last place). The bound is 4 u^2 / |x|
(u = 2^-24): with x in [1, 2) the word e = 1 - x r0 is at most 1.5 u, and four
quantities of at most that size are rounded once, each by u^2 at most (relative
to 1 / x). Non-finite seeds come back as they are."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "nalu-wind_gb300" / "csrc"


@pytest.fixture(scope="module")
def rcp(tmp_path_factory):
    so = tmp_path_factory.mktemp("dd_rcp") / "libdd_rcp.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(so),
                    str(HERE / "dd_rcp_host.cpp")], check=True)
    f = ctypes.CDLL(str(so)).dd_rcp_seeded

    def call(hi, lo, seed):
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        out = np.empty_like(hi), np.empty_like(hi)
        f(ctypes.c_int64(hi.size), p(hi), p(lo), p(seed), p(out[0]), p(out[1]))
        return out
    return call


@pytest.mark.parametrize("off", [0.0, 2.0 ** -24, -2.0 ** -24, 2.0 ** -23, -2.0 ** -23, 2.0 ** -22, -2.0 ** -22, 2.0 ** -21,
                                 -2.0 ** -21])
def test_error_for_seeds_off_by(rcp, off):
    rng = np.random.default_rng(5)
    n = 1 << 19
    x = rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * 2.0 ** rng.integers(-40, 40, n)
    hi = x.astype(np.float32)
    lo = (x - hi.astype(np.float64)).astype(np.float32)
    seed = ((1 + off) / hi.astype(np.float64)).astype(np.float32)
    r = rcp(hi, lo, seed)
    X = hi.astype(np.longdouble) + lo.astype(np.longdouble)
    err = np.abs((r[0].astype(np.longdouble) + r[1].astype(np.longdouble)) * X - 1)
    assert err.max() <= 4 * 2.0 ** -48


def test_special_seeds(rcp):
    hi = np.array([0.0, -0.0, np.inf, np.nan], np.float32)
    with np.errstate(divide="ignore", invalid="ignore"):
        r = rcp(hi, np.zeros_like(hi), np.array([np.inf, -np.inf, np.inf, np.nan], np.float32))
    np.testing.assert_array_equal(r[0], np.array([np.inf, -np.inf, np.inf, np.nan], np.float32))
