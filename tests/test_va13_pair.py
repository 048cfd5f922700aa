"""minfor's two rank-one updates of a step side by side (mc11a_pair_w) against
mc11a called twice: the same bits for random factors and vectors, with
diagonal entries that are not positive, zero and NaN elements, and scalars
over the whole range for which the pair form is taken."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def pair(tmp_path_factory):
    out = tmp_path_factory.mktemp("va13") / "libva13pair.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    str(HERE / "csrc" / "va13_pair.cpp"), "-o", str(out)], check=True)
    f = C.CDLL(str(out)).va13_update_pair
    f.argtypes = [C.c_int] + [C.c_void_p] * 4 + [C.c_double] * 2 + [C.c_void_p] * 2
    return f


@pytest.mark.parametrize("n", [2, 3, 6, 15, 16])
def test_pair_equals_two_updates(pair, n):
    rng = np.random.default_rng(n)
    na = n * (n + 1) // 2
    diag = np.cumsum([0] + [n - i for i in range(n - 1)])
    for trial in range(3000):
        a = rng.normal(0, 1, na)
        a[diag] = np.abs(a[diag]) + 0.1
        if trial % 3 == 0:
            k = rng.integers(n)
            a[diag[k]] = rng.choice([0.0, -0.0, -1.0, np.nan])
        v = [rng.normal(0, 1, n) for _ in range(3)]
        if trial % 4 == 0:
            v[rng.integers(3)][rng.integers(n)] = rng.choice([0.0, np.nan, np.inf])
        dga, den = -float(rng.lognormal(0, 3)), float(rng.lognormal(0, 3))
        if trial % 50 == 0:
            dga = float(rng.choice([-5e-324, -1.7976931348623157e308]))
        if trial % 70 == 0:
            den = float(rng.choice([5e-324, 1.7976931348623157e308]))
        o1, o2 = np.zeros(na + n + 1), np.zeros(na + n + 1)
        assert pair(n, a.ctypes.data, v[0].ctypes.data, v[1].ctypes.data, v[2].ctypes.data, dga, den,
                    o1.ctypes.data, o2.ctypes.data) == 0
        assert np.array_equal(o1, o2, equal_nan=True)
