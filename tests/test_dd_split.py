"""The splits of a double into a float pair (dd.h), on the host: the plain
split keeps 48 bits, the nearest one 49 with |lo| <= ulp(hi) / 2, and the
variants for zeros and triples give the plain split, for ordinary values,
powers of two and their neighbours, zeros, values at the ends of the integer
path (2^-62, 2^127) and non-finite ones."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    exe = tmp_path_factory.mktemp("dd") / "dd_split"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "nalu-wind_gb300" / "csrc"),
                    str(ROOT / "tests" / "dd_split_host.cpp"), "-o", str(exe)], check=True)

    def run(x):
        r = subprocess.run([str(exe)], input=x.tobytes(), capture_output=True, check=True)
        return np.frombuffer(r.stdout, np.float32).reshape(4, len(x), 2)
    return run


def _ordinary():
    rng = np.random.default_rng(3)
    m = rng.uniform(1.0, 2.0, 30000) * 2.0 ** rng.integers(-62, 127, 30000) * rng.choice([-1.0, 1.0], 30000)
    p = 2.0 ** np.arange(-61, 127, dtype=np.float64)
    near = np.concatenate([np.nextafter(p, 0), p, np.nextafter(p, np.inf), p * (1 + 2.0 ** -24),
                           p * (2 - 2.0 ** -25), p * (2 - 2.0 ** -52)])
    x = np.concatenate([m, near, -near])
    return x[: len(x) // 3 * 3]


def test_ordinary_values(splits):
    x = _ordinary()
    plain, z, near, three = splits(x)
    np.testing.assert_array_equal(plain, z)
    np.testing.assert_array_equal(plain, three)
    back = plain.astype(np.float64).sum(1)  # exact in FP64: 48 or 49 bits
    assert np.all(np.abs(back - x) <= 2.0 ** -48 * np.abs(x))
    nb = near.astype(np.float64).sum(1)
    assert np.all(np.abs(nb - x) <= 2.0 ** -49 * np.abs(x))
    ulp = np.spacing(np.abs(near[:, 0])).astype(np.float64)
    assert np.all(np.abs(near[:, 1].astype(np.float64)) <= 0.5 * ulp)


def test_zeros_small_large_and_non_finite(splits):
    x = np.array([0.0, -0.0, 1.0, 2.0 ** -62, 2.0 ** -63, -2.0 ** -70, 2.0 ** 127, -3e38, 2.0 ** -126, np.inf, -np.inf, 0.0])
    with np.errstate(over="ignore"):
        plain, z, near, three = splits(x)
    np.testing.assert_array_equal(plain, three)
    np.testing.assert_array_equal(plain, z)
    for s in (plain, near):
        np.testing.assert_array_equal(s[:2], 0.0)
        fin = np.isfinite(x)
        assert np.all(np.abs(s[fin].astype(np.float64).sum(1) - x[fin]) <= 2.0 ** -47 * np.abs(x[fin]))
        assert s[9, 0] == np.inf and s[10, 0] == -np.inf
    nan = splits(np.array([np.nan, 1.0, np.nan]))
    assert np.isnan(nan[0][0, 0]) and np.isnan(nan[2][0, 0]) and np.isnan(nan[3][2, 0]) and nan[3][1, 0] == 1.0
