"""The search by sums over bins (search_packet 0) against the packet kernels,
whose per-lane sums run in the reference's order: the same requests and the
same number of acceptance tests, in both precision forms.  The cases are where
it can go wrong: two to nine neurons, networks whose leaves lie as deep as the
keys allow, types without vacant dendrites (every search fails), totals that
underflow or are zero (left to the ordered form), the kernels that need the
distance itself, small acceptance criteria, and batched contexts."""
import numpy as np
import pytest

import relearn_b200 as R
from relearn_b200 import workloads as W

pytestmark = pytest.mark.gpu

PACKETS, BINS = dict(search_warps=2, search_packet=32, search_cap=1), dict(search_warps=4, search_packet=0, search_cap=0)


def both(net, axons, exc, inh, signal, step=3):
    out = []
    for shape in (PACKETS, BINS):
        net.set_tuning(**shape)
        net.prepare_update_connectivity(axons, exc, inh, signal=signal)
        before = net.stats()["nodes_touched"]
        out.append((net.find_targets(step), net.stats()["nodes_touched"] - before))
    return out


def network(n, precision, positions=None, side=None, **change):
    side = side or (1000.0 * n) ** (1.0 / 3.0)
    p = R.default_params(n, side)
    p.update(precision=precision, seed=11, **change)
    net = R.Network(p)
    sig = W.signal_types(n, 3) if n > 4 else np.arange(n, dtype=np.uint8) % 2
    net.set_positions(W.uniform_cube(n, side, 3) if positions is None else positions, sig)
    return net, sig


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["2", "3", "9", "33", "4001", "deep", "mixture", "no_inh", "none", "underflow", "far", "cutoff", "linear", "gamma",
                                  "weibull", "mu", "theta_small", "theta_half", "sparse", "several_axons"])
def test_bins_equal_packets(case, precision):
    rng = np.random.default_rng(7)
    n, change, pos = 2500, {}, None
    if case.isdigit():
        n = int(case)
    elif case == "deep":  # pairs a few 1e-9 um apart: leaves more than 30 levels below the root
        n = 600
        pos = W.uniform_cube(n, 800.0, 5)
        pos[1::2] = pos[0::2] + 3e-9
        pos = np.clip(pos, 0.0, 799.9)
        change["side"] = 800.0
    elif case == "mixture":
        pos = W.gaussian_mixture(n, 3000.0, 5, components=8, std=20.0)
        change["side"] = 3000.0
    elif case == "underflow":
        change["sigma"] = 0.2
    elif case == "far":
        change["sigma"] = 1.5
    elif case in ("cutoff", "linear"):
        change.update(kernel_type=R.KERNEL_LINEAR, linear_cutoff=4.0 if case == "cutoff" else 300.0)
    elif case == "gamma":
        change.update(kernel_type=R.KERNEL_GAMMA, kernel_k=2.0, kernel_scale=300.0)
    elif case == "weibull":
        change.update(kernel_type=R.KERNEL_WEIBULL, kernel_k=2.0, kernel_scale=1e-5)
    elif case == "mu":
        change["mu"] = 120.0
    elif case == "theta_small":
        change["theta"] = 0.05
    elif case == "theta_half":
        change["theta"] = 0.5
    net, sig = network(n, precision, pos, **change)
    axons = np.ones(n, np.uint32)
    exc, inh = np.ones(n, np.uint32), np.ones(n, np.uint32)
    if case == "no_inh":
        inh[:] = 0
    elif case == "none":
        exc[:] = 0
        inh[:] = 0
        exc[5] = 1  # one target: it finds nothing itself
    elif case == "sparse":
        axons[:] = 0
        axons[rng.permutation(n)[:7]] = 1
        exc = (rng.random(n) < 0.05).astype(np.uint32)
    elif case == "several_axons":
        axons = rng.integers(0, 4, n).astype(np.uint32)
        exc = rng.integers(0, 3, n).astype(np.uint32)
    (a, ta), (b, tb) = both(net, axons, exc, inh, sig)
    assert np.array_equal(a, b)
    if precision == 0 and case not in ("underflow", "far", "cutoff"):
        assert ta == tb  # the packets count a second, distance-weighted walk where a total is 0
    net.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_bins_equal_packets_in_an_ensemble(precision):
    nets = [dict(num_neurons=k, seed=40 + i, side=(1000.0 * k) ** (1 / 3), theta=t, sigma=s, growth_rate=1e-4)
            for i, (k, t, s) in enumerate([(1, 0.3, 750.0), (700, 0.2, 500.0), (2, 0.3, 750.0), (333, 0.5, 1000.0), (1500, 0.3, 90.0)])]
    base = R.default_params(1, 1.0)
    base["precision"] = precision
    net = R.Network(base, networks=nets)
    sig = np.concatenate([W.signal_types(d["num_neurons"], 2) for d in nets])
    net.set_positions(np.concatenate([W.uniform_cube(d["num_neurons"], d["side"], 9 + i) for i, d in enumerate(nets)]), sig)
    one = np.ones(net.n, np.uint32)
    (a, _), (b, _) = both(net, one, one, one, sig)
    assert len(a) > 2000 and np.array_equal(a, b)
    net.close()
