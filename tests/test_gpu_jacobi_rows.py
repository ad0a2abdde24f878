"""Jacobi-PCG in registers (systems of 64 rows and more) with rows around and far above the five entries
a thread keeps: the rest of a row is read from memory.  The general kernel solves the same systems."""
import numpy as np
import pytest
from test_gpu_assembly import fan_network
from test_gpu_jacobi_sizes import solve

from cicy_geom_b200.network import HostNetwork, NetworkConfig

pytestmark = pytest.mark.gpu


def comb(rungs):
    """Two spines; every third rung site has one rung, a second rung below it, and also a stub: spine
    nodes of four, five and six entries."""
    length = max(0.02 * rungs + 0.1, 1.0)
    cfg = NetworkConfig(side=length, n_cnts=1, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0), gs_min=max(0.05, length / 60))
    cnts = []
    for y, lo, hi in ((0.25, -0.04, length - 0.05), (0.75, 0.05, length + 0.04)):
        x = np.arange(round(lo * 100), round(hi * 100) + 1) / 100
        cnts.append(np.stack([x, np.full(len(x), y), np.full(len(x), 0.5)], 1))
    y = np.arange(25, 76) / 100
    for k in range(rungs):
        x, lift = 0.06 + 0.02 * k, 0.0108 + 1e-5 * (k % 7)
        for z in (0.5 + lift, 0.5 - lift)[:1 + (k % 3 > 0)]:
            cnts.append(np.stack([np.full(len(y), x), y, np.full(len(y), z)], 1))
        if k % 3 == 2:
            stub = 0.25 - lift - np.arange(10) / 100
            cnts.append(np.stack([np.full(10, x), stub, np.full(10, 0.5)], 1))
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cnts])])
    xyz, n = np.concatenate(cnts), len(cnts)
    return cfg, HostNetwork.from_arrays({
        "x": xyz[:, 0], "y": xyz[:, 1], "z": xyz[:, 2], "flag": np.repeat(np.arange(n), np.diff(ptr)), "structure_ptr": ptr,
        "structure_idx": np.arange(len(xyz)), "radii": np.full(n, cfg.radius), "window": [0, 0, 0] + 6 * [length]}).extract_window(cfg)


def check(net, cfg):
    """Agreement of the two kernels; entries of each row of the unit-resistor system."""
    fast, r_fast, S = solve(net, cfg, True)
    general, r_general, _ = solve(net, cfg, False)
    assert [s[0] for s in fast] == [s[0] for s in general] and fast[0][2] == 1 and all(s[2] == 0 for s in general)
    assert all(s[1] <= 1e-10 for s in fast + general)
    assert 0 < r_general < 1e18 and abs(r_fast - r_general) <= 1e-9 * r_general
    n = len(S["diag"])
    assert n >= 64
    return 1 + np.diff(S["row_ptr"]) + np.bincount(S["col_ind"], minlength=n)


@pytest.mark.parametrize("rungs", [15, 60, 200, 700])  # one CTA with one and several rows a thread, two and four
def test_rows_of_four_to_six_entries(cuda_ok, rungs):
    cfg, net = comb(rungs)
    entries = np.bincount(check(net, cfg), minlength=8)
    assert entries[4] > 0 and entries[5] > 0 and entries[6] > 0 and not entries[7:].any()


@pytest.mark.parametrize("spokes", [70, 300, 2100])  # one CTA, one with two rows a thread, a cluster
def test_long_row(cuda_ok, spokes):
    cfg = NetworkConfig(side=1.0, n_cnts=spokes + 1, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0))
    assert check(fan_network(spokes, cfg), cfg).max() > spokes
