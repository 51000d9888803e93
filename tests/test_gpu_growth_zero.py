"""A growth curve whose two ends coincide at zero (minimum and target calcium
0): a neuron with calcium 0 neither grows nor retracts, whatever the zeros'
signs, in every kernel that runs the curve."""
import numpy as np
import pytest

from conftest import small_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("minimum,target", [(0.0, 0.0), (-0.0, 0.0), (-0.0, -0.0), (0.0, -0.0)])
@pytest.mark.parametrize("synapses,fused", [(False, True), (True, True), (True, False)])
def test_flat_curve_at_zero(synapses, fused, minimum, target, precision):
    from relearn_b200 import Network

    n = 900
    params, pos, sig = small_network(n, 900.0, 3)
    params.update(precision=precision, min_calcium=(minimum,) * 3, target_calcium=target, noise_mean=0.0, noise_stddev=0.1)
    net = Network(params)
    net.set_positions(pos, sig)
    if synapses:
        net.add_edges(np.arange(n), np.roll(np.arange(n), 1), np.ones(n, np.int32))
    net.set_step_fusion(fused)
    net.activity_block(1, 20)
    state = net.neurons()
    assert not state["fired"].any() and not state["calcium"].any()
    for t in range(3):
        assert not net.get_elements(t)["delta"].any()
    net.close()
