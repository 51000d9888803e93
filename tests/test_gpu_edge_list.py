"""rl_get_edges: equal pairs aggregated, pairs that sum to zero left out,
whatever the runs' lengths, and any part of the list into any of the arrays."""
import ctypes as C

import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W

pytestmark = pytest.mark.gpu


def network(n=300):
    net = R.Network(R.default_params(n, 700.0))
    net.set_positions(W.uniform_cube(n, 700.0, 5), W.signal_types(n, 5))
    return net


def aggregated(t, s, w):
    key = t.astype(np.uint64) << 32 | s
    pair, where = np.unique(key, return_inverse=True)
    total = np.zeros(len(pair), np.int64)
    np.add.at(total, where, w)
    keep = total != 0
    return (pair[keep] >> 32).astype(np.uint32), pair[keep].astype(np.uint32), total[keep].astype(np.int32)


# runs around the share of one thread, of a warp's pass, and across thread blocks
@pytest.mark.parametrize("lengths", [[1], [1, 2, 1], [31, 32, 33, 34, 1], [159, 160, 161, 162, 3, 1], [5000, 1, 5000], [33] * 40, [257, 255, 256]])
@pytest.mark.parametrize("zero", [False, True])
def test_runs_of_equal_pairs(lengths, zero):
    rng = np.random.default_rng(len(lengths))
    net = network()
    pairs = rng.permutation(300 * 300)[: len(lengths)]
    t = np.repeat(pairs // 300, lengths).astype(np.uint32)
    s = np.repeat(pairs % 300, lengths).astype(np.uint32)
    w = rng.integers(-4, 5, len(t)).astype(np.int32)
    if zero:  # every other run sums to zero
        ends = np.cumsum(lengths)
        for k in range(0, len(lengths), 2):
            w[ends[k] - 1] -= w[ends[k] - lengths[k] : ends[k]].sum()
    order = rng.permutation(len(t))
    net.add_edges(t[order], s[order], w[order])
    for got, want in zip(net.edges(), aggregated(t, s, w)):
        assert np.array_equal(got, want)
    net.close()


def test_capacity_and_missing_arrays():
    rng = np.random.default_rng(4)
    net = network()
    m = 4000
    t, s = (rng.integers(0, 300, m).astype(np.uint32) for _ in range(2))
    w = rng.integers(-2, 3, m).astype(np.int32)
    net.add_edges(t, s, w)
    want = aggregated(t, s, w)
    k = len(want[0])
    for capacity in (0, 1, 17, k - 1, k, k + 5):
        for given in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 0)):
            out = [np.full(capacity + 1, 77, d) if g else None for g, d in zip(given, (np.uint32, np.uint32, np.int32))]
            count = C.c_uint64()
            assert net.lib.rl_get_edges(net.h, *(None if a is None else a.ctypes.data_as(C.c_void_p) for a in out), capacity, C.byref(count)) == 0
            assert count.value == k
            for a, b in zip(out, want):
                if a is not None:
                    assert np.array_equal(a[: min(k, capacity)], b[:capacity]) and (a[min(k, capacity):] == 77).all()
    net.close()
    empty = network()
    assert all(len(a) == 0 for a in empty.edges())
    empty.close()
