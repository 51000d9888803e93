"""FP32 blocks of steps without synapses on both sides of the size from which a
thread takes a neuron pair: the bits of one launch per step, at an odd last
pair, with disabled neurons and with targets of their own."""
import numpy as np
import pytest

from test_gpu_fusion import assert_same, make, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [249_999, 250_000, 250_001, 250_177])
@pytest.mark.parametrize("mode", ["all", "disabled", "targets"])
def test_pairs_equal_steps(n, mode):
    runs = []
    for fused in (True, False):
        net = make(n, 31, 1)
        net.set_step_fusion(fused)
        if mode == "disabled":
            net.set_enabled((np.random.default_rng(3).random(n) > 0.25).astype(np.uint8))
            net.set_neurons(fired=(np.random.default_rng(6).random(n) < 0.3).astype(np.uint8))
        elif mode == "targets":
            net.set_target_calcium(np.random.default_rng(4).uniform(0.0, 0.9, n))
        got = []
        for first, count in ((1, 37), (38, 64), (102, 2)):
            net.activity_block(first, count)
            got.append(state(net))
        runs.append(got)
        net.close()
    for i, (a, b) in enumerate(zip(*runs)):
        assert_same(a, b, (mode, i))
    assert any(st["fired"].any() for st in runs[0])
