"""Which kernels a search list takes: the bins form settles an ordinary list by
itself; what it leaves open goes to the ordered form, one search per warp or,
where a large share of a dense list is open, in packets; and what does not fit
a warp's scratch goes to the packets behind that.  Requests and acceptance
tests are those of the packets alone on every route."""
import numpy as np
import pytest

import relearn_b200 as R
from test_gpu_search_bins import BINS, PACKETS, network

pytestmark = pytest.mark.gpu


def run(net, shape, axons, one, sig):
    """Requests, acceptance tests and launches of one search."""
    net.set_tuning(**shape)
    net.prepare_update_connectivity(axons, one, one, signal=sig)
    net.find_targets(2)  # buffers are grown by now, octree records packed
    a = net.stats()
    req = net.find_targets(3)
    b = net.stats()
    return req, b["nodes_touched"] - a["nodes_touched"], b["gpu_launches"] - a["gpu_launches"]


# launches behind those of a search in packets (one per signal type): the bins
# form alone is one less, the ordered form and a packet launch per signal type
# come on top
ROUTES = {"bins": -1, "ordered": 0, "packets": 1, "ordered, then packets": 2}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case,n,change,share,route", [
    ("ordinary", 9, {}, 1.0, "bins"),
    ("ordinary", 33, {}, 1.0, "bins"),
    ("ordinary", 2500, {}, 0.01, "bins"),
    ("underflow", 2500, dict(sigma=0.2), 1.0, "ordered"),
    ("far", 2500, dict(sigma=1.5), 1.0, ("bins", "ordered")),  # weights below FP32's range, not FP64's
    ("cutoff", 2500, dict(kernel_type=R.KERNEL_LINEAR, linear_cutoff=4.0), 1.0, "ordered"),
    ("underflow, many", 20000, dict(sigma=0.2), 1.0, "ordered"),
    ("underflow, more", 64000, dict(sigma=0.2), 1.0, ("ordered", "packets")),
    ("underflow, most", 290000, dict(sigma=0.1), 1.0, "packets"),
    ("underflow, sparse", 20000, dict(sigma=0.2), 0.01, "ordered"),
    ("long walks", 20000, dict(sigma=0.2, theta=0.05), 0.02, "ordered, then packets"),
])
def test_route(case, n, change, share, route, precision):
    net, sig = network(n, precision, **change)
    rng = np.random.default_rng(n)
    axons = (rng.random(n) < share).astype(np.uint32)
    axons[[int(np.argmax(sig == 0)), int(np.argmax(sig == 1))]] = 1
    one = np.ones(n, np.uint32)
    a, ta, la = run(net, PACKETS, axons, one, sig)
    b, tb, lb = run(net, BINS, axons, one, sig)
    assert np.array_equal(a, b)
    assert ta == tb
    assert lb - la == ROUTES[route if isinstance(route, str) else route[precision]]
    net.close()
