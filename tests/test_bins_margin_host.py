"""The margin within which the FP32 search by bins does not trust its own order
of additions: at least what the ordered sums can differ by, for every number of
visited nodes that an octree can have."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
U = 2.0**-24


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "bins_margin_probe.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "helpers", "bins_margin_probe.cpp")], check=True)
    lib = C.CDLL(so)
    lib.probe_margin.restype, lib.probe_margin.argtypes = C.c_double, [C.c_double, C.c_uint32]
    lib.probe_kahan.restype, lib.probe_kahan.argtypes = C.c_float, [C.c_long, C.c_void_p]
    return lib


@pytest.mark.parametrize("n", [1, 1000, 10**5, 10**6, 4_500_000, 10**8, 2**32 - 1])
def test_margin_covers_both_sums_and_the_threshold(probe, n):
    kahan = 2 * U + 8 * n * U * U  # the running sum, and the total behind r
    assert probe.probe_margin(1.0, n) >= 2 * kahan + U + 2 * n * 2.0**-53
    assert probe.probe_margin(3.0, n) == 3.0 * probe.probe_margin(1.0, n)


@pytest.mark.parametrize("kind", ["uniform", "wide", "equal", "descending"])
def test_compensated_sum_is_within_its_share(probe, kind):
    rng = np.random.default_rng(3)
    n = 1 << 22
    x = {"uniform": rng.random(n), "wide": np.exp(rng.uniform(-40, 0, n)), "equal": np.full(n, 0.1), "descending": 1.0 / np.arange(1, n + 1)}[kind]
    x = np.ascontiguousarray(x, np.float32)
    exact = math.fsum(x.tolist())
    assert abs(probe.probe_kahan(n, x.ctypes.data) - exact) <= (2 * U + 8 * n * U * U) * exact
