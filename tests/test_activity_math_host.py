"""The activity kernels' rearranged arithmetic against the step-by-step
formulas, bit for bit, on the host (the GPU parity tests compare whole runs
with the oracle)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "activity_math_probe.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-mfma", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "helpers", "activity_math_probe.cpp")], check=True)
    lib = C.CDLL(so)
    for f in (lib.probe_curve, lib.probe_uniform):
        f.restype = C.c_long
        f.argtypes = [C.c_long, C.c_void_p]
    return lib


def test_growth_curve_exponential(probe):
    rng = np.random.default_rng(4)
    edges = [0.0, 5e-324, 1e-300, 739.9999999, 740.0, 740.0000001, 745.2, 746.0, 1e5, 1e300, float("inf"), float("nan")]
    k = np.arange(0, 64 * 800) * (np.log(2.0) / 64.0)  # where the table index steps
    q = np.concatenate([edges, rng.uniform(0, 3, 400_000), rng.uniform(0, 760, 200_000), 10.0 ** rng.uniform(-20, 4, 100_000),
                        k, np.nextafter(k, 0), np.nextafter(k, 1e9), k + np.log(2.0) / 128.0])
    q = np.ascontiguousarray(np.abs(q))
    assert probe.probe_curve(len(q), q.ctypes.data) == 0


def test_uniform_without_conversion(probe):
    rng = np.random.default_rng(5)
    top = 1 << 52
    lo, hi = int(0.075 * 2.0**53), int(0.925 * 2.0**53)
    edges = np.concatenate([np.arange(0, 4096), np.arange(top - 4096, top + 4096), np.arange(2 * top - 4096, 2 * top),
                            np.arange(lo - 4096, lo + 4096), np.arange(hi - 4096, hi + 4096)]).astype(np.uint64)
    b = np.concatenate([edges, rng.integers(0, 2 * top, 1_000_000, dtype=np.uint64)])
    assert probe.probe_uniform(len(b), b.ctypes.data) == 0
