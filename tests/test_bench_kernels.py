"""bench.py names the kernel that ran: the route of a join from the launches and
phases it reports, and DRAM traffic only where that kernel was captured."""
import pytest

import bench


@pytest.mark.parametrize("algo,kernels,phases,route", [
    ("PRO", 1, (0, 0, 0, .01), "small"),
    ("NPO", 1, (0, 0, 0, .01), "small"),
    ("NPO", 2, (0, .05, 0, .07), "table"),
    ("NPO", 4, (.1, .05, 0, .07), "regions"),
    ("NPO", 4, (.1, 0, .01, .1), "hashed, one pass"),
    ("NPO", 8, (.9, 1., .01, .9), "hashed"),
    ("PRO", 4, (.05, 0, .01, .04), "radix, one pass"),
    ("PRHO", 8, (.9, 1., .01, .7), "radix"),
    ("m-way", 4, (.05, 0, .01, .04), "sorted, one pass"),
    ("m-pass", 8, (.9, 1., .01, 1.2), "sorted"),
])
def test_route(algo, kernels, phases, route):
    assert bench.route_of(algo, kernels, phases) == route
    kernel = bench.KERNELS[route]
    dom = max(kernel, key=lambda k: phases[k])
    assert phases[dom] == max(phases)      # the phase that took longest has its kernel
    name, _, traffic = kernel[dom]
    assert traffic is None or route in ("radix", "sorted")
    assert ("hashed" in name or "sorted" in name or "npo" in name) == (algo[0] != "P" and kernels > 1)
