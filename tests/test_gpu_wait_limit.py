"""A block of steps whose wait between two steps runs out: the kernel returns,
the next call that waited for it says so under its own name, and the context
refuses everything from then on, while others go on."""
import numpy as np
import pytest

import relearn_b200 as R
from conftest import small_network

pytestmark = pytest.mark.gpu

RL_ERR_TIMEOUT = 4
# one neuron per thread, and several (both precision forms: more than 170,496)
SIZES = [20_011, 180_001]


def network(n, precision, edges=1):
    params, pos, sig = small_network(n, 2500.0, 11)
    params["precision"] = precision
    net = R.Network(params)
    net.set_positions(pos, sig)
    rng = np.random.default_rng(n)
    net.add_edges(rng.integers(0, n, edges), rng.integers(0, n, edges), np.ones(edges, np.int32))
    return net


READS = {
    "neurons": lambda net: net.neurons(),
    "elements": lambda net: net.get_elements(0),
    "edges": lambda net: net.edges(),
    "stats": lambda net: net.stats(),
    "synchronize": lambda net: net.synchronize(),
    "snapshot": lambda net: (net.snapshot_neurons(np.zeros(net.n)), net.snapshot_wait()),
    "update": lambda net: net.plasticity_update(100),
    "simulate": lambda net: net.simulate(101, 200),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("read", sorted(READS))
def test_lost_block_is_reported_and_stays_refused(read, n, precision):
    net = network(n, precision)
    net.activity_block(1, 20)
    before = net.neurons()
    assert np.isfinite(before["x"]).all()
    net.set_wait_limit(1)  # every block but the last to arrive gives up at its first wait
    net.activity_block(21, 80)
    with pytest.raises(R.RelearnError) as e:
        READS[read](net)
    assert e.value.status == RL_ERR_TIMEOUT and "barrier between steps" in str(e.value)
    for call in list(READS.values()) + [lambda net: net.activity_block(101, 2), lambda net: net.set_wait_limit(0), lambda net: net.tree()]:
        with pytest.raises(R.RelearnError) as e:
            call(net)
        assert e.value.status == RL_ERR_TIMEOUT
    net.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_other_contexts_go_on(precision):
    ref = network(SIZES[0], precision, 80_000)
    ref.set_step_fusion(False)
    ref.activity_block(1, 100)
    net = network(SIZES[0], precision, 80_000)
    lost = network(SIZES[1], precision)
    lost.set_wait_limit(1)
    lost.activity_block(1, 50)
    net.set_wait_limit(0)
    net.activity_block(1, 100)
    a, b = ref.neurons(), net.neurons()
    assert all(np.array_equal(a[k], b[k]) for k in a)
    with pytest.raises(R.RelearnError):
        lost.synchronize()
    lost.close()
    again = network(SIZES[1], precision)  # takes over the closed context's word
    again.activity_block(1, 50)
    again.synchronize()
    for net in (ref, net, again):
        net.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("hub", ["target", "source"])
def test_limit_leaves_room_for_a_neuron_with_every_synapse(hub, n, precision):
    """Its block walks the whole list by itself, tens of milliseconds, while
    the others wait; the limit set here is well below one."""
    net = network(n, precision)
    m = 600_000
    one, many = np.zeros(m, np.uint32), np.random.default_rng(2).integers(0, n, m).astype(np.uint32)
    net.add_edges(one if hub == "target" else many, one if hub == "source" else many, np.ones(m, np.int32))
    net.set_neurons(fired=np.ones(n, np.uint8))
    net.set_enabled((np.arange(n) > 0).astype(np.uint8) if hub == "source" else np.ones(n, np.uint8))  # keeps its spike flag
    net.set_wait_limit(100)
    net.activity_block(1, 4)
    net.synchronize()
    net.close()
