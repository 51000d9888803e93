"""A block of activity steps of a network with synapses in one launch gives the
bits of one launch per step: at the edges of its forms (a cluster of up to
sixteen blocks of 384 neurons, a resident grid of more, several neurons per
thread, one launch per step where even those do not hold the network), both precision forms, every neuron
model, disabled neurons that keep a set spike flag, targets of their own, other
substep counts, and blocks of even and odd length that follow each other."""
import numpy as np
import pytest

from conftest import small_network

pytestmark = pytest.mark.gpu

DRIVE = {0: {}, 1: dict(noise_mean=0.0, noise_stddev=0.1, conductance=0.3), 2: dict(noise_mean=0.7, noise_stddev=0.5, conductance=0.3),
         3: dict(noise_mean=600.0, noise_stddev=200.0, conductance=300.0)}


def make(n, precision, model, fused, h=10):
    from relearn_b200 import Network

    params, pos, sig = small_network(n, 2500.0, 11)
    params.update(precision=precision, neuron_model=model, h_model=h, **DRIVE[model])
    net = Network(params)
    net.set_positions(pos, sig)
    rng = np.random.default_rng(n)
    m = 6 * n
    # sources crowd together: rows of very different length, a target hit by many
    src = (n * rng.random(m) ** 3).astype(np.uint32)
    tgt = (n * rng.random(m) ** 2).astype(np.uint32)
    net.add_edges(tgt, src, rng.choice(np.array([-3, -1, 1, 2, 5], np.int32), m))
    net.set_enabled((rng.random(n) > 0.2).astype(np.uint8))
    net.set_neurons(fired=(rng.random(n) < 0.3).astype(np.uint8))
    if n % 2:
        net.set_target_calcium(rng.uniform(0.3, 0.9, n))
    net.set_step_fusion(fused)
    return net


def state(net):
    out = dict(net.neurons())
    for t in range(3):
        out[f"delta{t}"] = net.get_elements(t)["delta"]
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,model,h", [(2, 0, 10), (383, 0, 10), (384, 0, 7), (385, 1, 10), (3073, 0, 10), (6144, 0, 10), (6145, 0, 10), (6145, 3, 10), (6144, 3, 10),
                                       (20011, 0, 10), (20012, 0, 10), (20011, 2, 10), (20012, 1, 10), (113664, 0, 10), (113665, 0, 10),
                                       (170496, 0, 10), (170497, 0, 10), (180001, 3, 10), (180002, 1, 10), (180003, 2, 10), (180004, 0, 7),
                                       (400003, 0, 10), (1136640, 0, 10), (1136641, 0, 10)])
def test_coupled_block_equals_steps(n, model, h, precision):
    nets = [make(n, precision, model, fused, h) for fused in (False, True)]
    spikes = 0
    for first, count in ((1, 37), (38, 1), (39, 2), (41, 100)):
        for net in nets:
            net.activity_block(first, count)
            net.synchronize()
        a, b = (state(net) for net in nets)
        for k in a:
            assert np.array_equal(a[k].view(np.uint8), b[k].view(np.uint8)), (first, k)
        spikes += int(a["fired"].sum())
    assert spikes > 0 or n < 100
    for net in nets:
        net.close()
