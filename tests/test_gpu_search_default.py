"""The search shape without tuning, on both sides of each line of its rule, and
that it finds what the other shape finds.  A shape that the caller or the tuner
set stays."""
import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W
from test_gpu_search_bins import BINS, PACKETS

pytestmark = pytest.mark.gpu

GAMMA = dict(kernel_type=R.KERNEL_GAMMA, kernel_k=2.0, kernel_scale=375.0)
LINEAR = dict(kernel_type=R.KERNEL_LINEAR, linear_cutoff=300.0)


@pytest.mark.parametrize("precision,n,share,change,packet", [
    (0, 655_001, 1.0, {}, 0),
    (0, 655_001, 1.0, GAMMA, 32),
    (0, 655_001, 1.0, dict(mu=50.0), 32),
    (0, 645_001, 1.0, LINEAR, 0),
    (0, 900_001, 0.7, GAMMA, 0),
    (0, 100_003, 1.0, dict(theta=0.1), 0),
    (1, 555_001, 1.0, {}, 0),
    (1, 555_001, 1.0, dict(mu=50.0), 0),
    (1, 555_001, 1.0, LINEAR, 32),
    (1, 545_001, 1.0, GAMMA, 0),
    (1, 900_001, 0.7, GAMMA, 0),
    (1, 60_001, 1.0, dict(theta=0.11), 32),
    (1, 59_999, 1.0, dict(theta=0.11), 0),
    (1, 60_001, 1.0, dict(theta=0.16), 0),
    (1, 300_001, 1.0, dict(theta=0.16), 32),
    (1, 300_001, 1.0, dict(theta=0.17), 0),
])
def test_default_shape(precision, n, share, change, packet):
    side = (1000.0 * n) ** (1 / 3)
    net = R.Network(dict(R.default_params(n, side), precision=precision, **change))
    net.set_positions(W.uniform_cube(n, side, 5), W.signal_types(n, 5))
    axons = np.zeros(n, np.uint32)
    axons[: round(n * share)] = 1
    one = np.ones(n, np.uint32)
    net.prepare_update_connectivity(axons, one, one)
    got = net.find_targets(3)
    assert net.tuning()["search_packet"] == packet
    net.set_tuning(**(BINS if packet else PACKETS))
    assert np.array_equal(net.find_targets(3), got)
    assert net.tuning()["search_packet"] == (0 if packet else 32)
    net.close()
