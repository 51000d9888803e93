"""A plasticity update over synaptic elements that the synapse list does not
bear out (connected elements without synapses) is refused, whichever element
type they are of and whatever the passes after it do."""
import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W

pytestmark = pytest.mark.gpu

RL_ERR_DEVICE = 3


def network(precision, n=600):
    side = (1000.0 * n) ** (1 / 3)
    net = R.Network(dict(R.default_params(n, side), precision=precision))
    net.set_positions(W.uniform_cube(n, side, 5), np.zeros(n, np.uint8))
    return net


def retract(net, etype, neuron):
    """One connected element of the neuron whose growth takes it back."""
    n = net.n
    one = np.zeros(n)
    one[neuron] = 1.0
    net.set_elements(etype, one, -one, one.astype(np.uint32), np.zeros(n, np.uint32))


def refused(net, step):
    with pytest.raises(R.RelearnError) as e:
        net.plasticity_update(step)
    assert e.value.status == RL_ERR_DEVICE and "synapse deletion" in str(e.value)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("etype", [0, 1, 2])
def test_elements_without_synapses(etype, precision):
    net = network(precision)
    retract(net, etype, 17)
    refused(net, 100)
    net.plasticity_update(200)  # reported once; the elements are gone
    net.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_elements_left_behind_by_an_emptied_list(precision):
    net = network(precision)
    net.load_network([3], [5], [1])
    retract(net, 0, 5)
    net.plasticity_update(100)
    assert net.stats()["synapses_deleted"] == 1 and len(net.edges()[0]) == 0
    for etype in range(3):
        retract(net, etype, 5)
        refused(net, 200 + 100 * etype)
    net.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_deletions_before_the_refusal_are_counted(precision):
    """The axon pass deletes the one synapse; the dendrite pass then finds one
    element more than synapses."""
    net = network(precision)
    net.load_network([3], [5], [1])
    retract(net, 0, 5)
    retract(net, 2, 8)
    refused(net, 100)
    assert net.stats()["synapses_deleted"] == 1 and net.stats()["bound_to_delete"] == 2
    assert len(net.edges()[0]) == 0
    net.close()
