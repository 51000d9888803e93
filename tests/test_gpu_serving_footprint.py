"""The admitted footprint bounds what a served run holds at its peak also when
the run searches from its first update on, from most of its neurons and at a
small theta, so that many of its searches are repeated in the reference's order
with scratch of their own."""
import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W
from relearn_b200.serving import Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,theta,axons", [(100_000, 0.15, (0.0, 4.0)), (300_000, 0.2, (1.0, 1.5))])
def test_peak_stays_below_the_footprint(n, theta, axons, precision):
    base = R.default_params(1, 1.0)
    base["precision"] = precision
    net = dict(num_neurons=n, seed=5, side=(1000.0 * n) ** (1 / 3), theta=theta, sigma=750.0, growth_rate=1e-4)
    pos, sig = W.request_inputs(net)
    grown = [g for g, _ in W.initial_elements(n, 7, *axons)]
    with Server(base, hbm_budget_bytes=60e9, slots=1, autotune=0) as srv:
        srv.submit(net, pos, sig, 201, grown=grown)
        done = []
        while not done:
            done = srv.poll(wait_ms=500)
    assert done[0]["status"] == 0 and done[0]["num_synapses"] > 0
    assert done[0]["device_peak_bytes"] <= done[0]["footprint_bytes"], done[0]["device_peak_bytes"] / done[0]["footprint_bytes"]
