"""The device generator takes 32, 8, 4, 2 or 1 threads per CNT by the number of CNTs;
each choice gives the host generator's network (counts and flags equal, coordinates to
the 1e-10 um the entry point promises)."""
from dataclasses import replace

import numpy as np
import pytest

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import NetworkConfig, generate_cnt_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1500, 1501, 6000, 6001, 12001, 30001])
@pytest.mark.parametrize("lengths", [(0.011, 0.05), (0.3, 0.4)])
def test_device_generator_against_host(cuda_ok, n, lengths):
    cfg = replace(NetworkConfig(side=2.0, n_cnts=n, seed=n), len_min=lengths[0], len_max=lengths[1])
    ref = generate_cnt_network(cfg).arrays()
    with Context(0) as ctx:
        ctx.generate_network(cfg, trim=False)
        got = ctx.network()
    assert np.array_equal(got["structure_ptr"], ref["structure_ptr"]) and np.array_equal(got["flag"], ref["flag"])
    assert np.array_equal(got["radii"], ref["radii"])
    for k in ("x", "y", "z"):
        assert np.max(np.abs(got[k] - ref[k])) < 1e-10
