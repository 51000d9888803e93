"""Contexts driven from different host threads at the same time: a kernel's
shared-memory limit belongs to the device, not to a context, so a context whose
octree is shallow, or whose network is small, must not take it away from one
that needs more between its setting and its launch."""
import threading

import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W

pytestmark = pytest.mark.gpu


def together(*work):
    """Runs the callables at the same time, one thread each; what they raised."""
    failed = []
    start = threading.Barrier(len(work))

    def one(f):
        start.wait()
        try:
            f()
        except Exception as e:
            failed.append(repr(e))

    threads = [threading.Thread(target=one, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return failed


def searcher(n, deep, precision):
    side = (1000.0 * n) ** (1 / 3)
    pos = W.uniform_cube(n, side, 5)
    if deep:  # pairs of neurons a few 1e-9 um apart: leaves more than 30 levels below the root
        pos[1::2] = np.clip(pos[0::2] + 3e-9, 0.0, 0.999 * side)
    net = R.Network(dict(R.default_params(n, side), precision=precision))
    net.set_positions(pos, W.signal_types(n, 5))
    axons = np.zeros(n, np.uint32)
    axons[:: max(1, n // 50)] = 1
    net.prepare_update_connectivity(axons, np.ones(n, np.uint32), np.ones(n, np.uint32))
    return net


@pytest.mark.parametrize("precision", [0, 1])
def test_searches_of_shallow_and_deep_octrees(precision):
    nets = [searcher(500, False, precision), searcher(600, True, precision), searcher(100_000, False, precision)]
    first = [net.find_targets(3) for net in nets]

    def loop(net, ref, times):
        for _ in range(times):
            assert np.array_equal(net.find_targets(3), ref)

    failed = together(*(lambda net=net, ref=ref, times=times: loop(net, ref, times) for net, ref, times in zip(nets, first, (12000, 12000, 3000))))
    assert not failed, failed[:3]
    assert all(len(r) for r in first)
    for net in nets:
        net.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_blocks_of_small_and_large_networks(precision):
    """Every block of steps stays one launch behind the descriptor's."""
    nets = []
    for n in (240_000, 900_001):  # several neurons per thread, in shared memory
        net = R.Network(dict(R.default_params(n, (1000.0 * n) ** (1 / 3)), precision=precision))
        rng = np.random.default_rng(n)
        net.set_positions(W.uniform_cube(n, (1000.0 * n) ** (1 / 3), 5), W.signal_types(n, 5))
        net.add_edges(rng.integers(0, n, n), rng.integers(0, n, n), np.ones(n, np.int32))
        net.activity_block(1, 3)
        net.synchronize()
        nets.append(net)
    before = [net.stats()["gpu_launches"] for net in nets]

    def loop(net):
        for k in range(6000):
            net.activity_block(4 + 3 * k, 3)
        net.synchronize()

    failed = together(*(lambda net=net: loop(net) for net in nets))
    assert not failed, failed[:3]
    assert [net.stats()["gpu_launches"] - b for net, b in zip(nets, before)] == [12000, 12000]
    for net in nets:
        net.close()
