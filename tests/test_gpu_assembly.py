"""Row assembly of the DEA systems where a node has many resistors: a fan of CNTs whose
junctions all sit on the end point of one CNT, at row lengths around the limits of the
row kernel (16 resistors held locally, insertion sort up to 32)."""
import math

import numpy as np
import pytest

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig
from oracle import cicy_oracle as O

pytestmark = pytest.mark.gpu


def fan_network(spokes, cfg):
    step, pts, ptr = 0.01, [], [0]

    def line(p0, p1):
        k = int(round(math.dist(p0, p1) / step))
        pts.extend(np.array(p0) + (np.array(p1) - np.array(p0)) * (i / k) for i in range(k + 1))
        ptr.append(len(pts))

    line((-0.045, 0.5, 0.5), (0.5, 0.5, 0.5))
    for k in range(spokes):
        t = 2 * math.pi * k / spokes
        u = np.array([0.3, math.cos(t), math.sin(t)]) / math.sqrt(1.09)
        line(tuple(np.array([0.5, 0.5, 0.5]) + 0.0105 * u), (1.045, 0.5 + 0.4 * math.cos(t), 0.5 + 0.4 * math.sin(t)))
    xyz, n = np.array(pts), len(ptr) - 1
    return HostNetwork.from_arrays({
        "x": xyz[:, 0], "y": xyz[:, 1], "z": xyz[:, 2], "flag": np.repeat(np.arange(n), np.diff(ptr)), "structure_ptr": ptr,
        "structure_idx": np.arange(len(xyz)), "radii": np.full(n, cfg.radius), "window": [0, 0, 0, 1, 1, 1, 1, 1, 1]}).extract_window(cfg)


@pytest.mark.parametrize("spokes", [13, 14, 15, 16, 30, 31, 32, 33, 70])
def test_fan_against_oracle(cuda_ok, spokes):
    cfg = NetworkConfig(side=1.0, n_cnts=spokes + 1, seed=0, tolerance=1e-14)
    net = fan_network(spokes, cfg)
    with Context(0) as ctx:
        ctx.upload(net)
        r = ctx.network_to_conductance(cfg.params())
        S = ctx.system(1)
    deg = np.diff(S["row_ptr"]) + np.bincount(S["col_ind"], minlength=len(S["diag"]))
    assert deg.max() >= spokes  # the fan's centre node
    ref = O.network_to_conductance(net.arrays(), O.params_from_config(cfg), solver="direct")
    np.testing.assert_allclose(np.array(r.resistances), ref["resistances"], rtol=1e-9)
