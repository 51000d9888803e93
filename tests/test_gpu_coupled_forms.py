"""Which form a block of steps with synapses takes, on both sides of each line:
one launch (a cluster, a resident grid, several neurons per thread) or one
launch per step, seen by the launches it makes.  (Their results are compared in
test_gpu_coupled.py; here the forms that its cases reach, and that they are
reached, for each precision form and model.)"""
import numpy as np
import pytest

import relearn_b200 as R
from conftest import small_network

pytestmark = pytest.mark.gpu

IZ, POISSON, FHN, AEIF = range(4)
ONE = 2  # the descriptor's launch and the block's


def launches(n, precision, model, steps, edges=None, fused=True):
    params, pos, sig = small_network(n, (1000.0 * n) ** (1 / 3), 11)
    params.update(precision=precision, neuron_model=model)
    net = R.Network(params)
    net.set_positions(pos, sig)
    m = edges or n
    k = np.arange(m, dtype=np.uint32) % n
    net.add_edges(k, (k + 1) % n, np.ones(m, np.int32))
    net.set_step_fusion(fused)
    net.activity_block(1, steps)
    before = net.stats()["gpu_launches"]
    net.activity_block(1 + steps, steps)
    net.synchronize()
    got = net.stats()["gpu_launches"] - before
    net.close()
    return got


@pytest.mark.parametrize("n,model,steps,form", [  # form: (FP64, FP32)
    (2, IZ, 7, "11"), (383, POISSON, 7, "11"), (6144, IZ, 7, "11"), (6145, AEIF, 7, "11"), (20_011, FHN, 2, "11"), (20_011, IZ, 1, "00"),
    (113_664, IZ, 2, "11"), (113_665, IZ, 2, "01"), (113_665, IZ, 3, "11"),
    (170_496, FHN, 4, "11"), (170_497, FHN, 4, "10"), (238_000, FHN, 4, "10"), (240_000, FHN, 4, "11"),
    (300_005, FHN, 4, "11"), (340_000, FHN, 4, "11"), (345_000, FHN, 4, "00"), (470_000, FHN, 4, "01"),
    (454_656, AEIF, 4, "11"), (454_657, AEIF, 4, "01"),
    (1_136_640, POISSON, 4, "11"), (1_136_641, IZ, 4, "01"), (1_875_456, IZ, 4, "01"), (1_875_457, IZ, 4, "00"),
])
@pytest.mark.parametrize("precision", [0, 1])
def test_form(n, model, steps, form, precision):
    got = launches(n, precision, model, steps)
    if form[precision] == "1":
        assert got == ONE
    else:
        assert got >= 1 + steps
    if n <= 20_011 and steps > 1:
        assert launches(n, precision, model, steps, fused=False) >= 1 + steps


@pytest.mark.parametrize("n,edges,one", [(120_001, 32_000_000, True), (120_001, 32_000_001, False), (113_001, 32_000_001, True)])
def test_long_lists_take_one_launch_per_step(n, edges, one):
    got = launches(n, 0, IZ, 4, edges)
    assert (got == ONE) if one else (got >= 5)
