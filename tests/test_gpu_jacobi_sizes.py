"""Jacobi-PCG around the sizes where its kernel changes: ladders of CNTs (two spines, rungs between
them) whose unit-resistor system has 6 rungs + 2 rows, and a fan whose centre row is longer than
the entries a thread keeps in registers.  The general (grid) kernel solves the same systems."""
import numpy as np
import pytest
from test_gpu_assembly import fan_network

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig

pytestmark = pytest.mark.gpu


def ladder(rungs):
    length, lines = max(0.02 * rungs + 0.1, 1.0), []
    cfg = NetworkConfig(side=length, n_cnts=rungs + 2, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0),
                        gs_min=max(0.05, length / 60))
    for y, lo, hi in ((0.25, -0.04, length - 0.05), (0.75, 0.05, length + 0.04)):
        x = np.arange(round(lo * 100), round(hi * 100) + 1) / 100
        lines.append(np.stack([x, np.full(len(x), y), np.full(len(x), 0.5)], 1))
    y = np.arange(20, 81) / 100
    lines += [np.stack([np.full(len(y), 0.06 + 0.02 * k), y, np.full(len(y), 0.5108 + 1e-5 * (k % 7))], 1) for k in range(rungs)]
    ptr = np.concatenate([[0], np.cumsum([len(v) for v in lines])])
    xyz, n = np.concatenate(lines), len(lines)
    return cfg, HostNetwork.from_arrays({
        "x": xyz[:, 0], "y": xyz[:, 1], "z": xyz[:, 2], "flag": np.repeat(np.arange(n), np.diff(ptr)), "structure_ptr": ptr,
        "structure_idx": np.arange(len(xyz)), "radii": np.full(n, cfg.radius), "window": [0, 0, 0] + 6 * [length]}).extract_window(cfg)


def solve(net, cfg, cluster):
    with Context(0) as ctx:
        ctx.set_solver(preconditioner=0, cluster=cluster)
        ctx.upload(net)
        r = ctx.network_to_conductance(cfg.params())
        return [(s.nodes, s.rel_residual, s.kernel) for s in r.solves[:r.n_solves]], r.resistances[0], ctx.system(0)


def check(net, cfg, rows):
    fast, r_fast, system = solve(net, cfg, True)
    general, r_general, _ = solve(net, cfg, False)
    assert len(system["diag"]) in rows
    assert [s[0] for s in fast] == [s[0] for s in general] and fast[0][2] == 1 and general[0][2] == 0
    assert all(s[1] <= 1e-10 for s in fast + general)
    assert 0 < r_general < 1e18 and abs(r_fast - r_general) <= 1e-9 * r_general


@pytest.mark.parametrize("edge", [70, 256, 512, 768, 1024, 1280, 1536, 2048, 3072, 4096, 6144, 8192, 12288])
@pytest.mark.parametrize("above", [0, 1])
def test_ladder(cuda_ok, edge, above):
    rungs = (edge - 2) // 6 + above
    cfg, net = ladder(rungs)
    check(net, cfg, range(edge - 5, edge + 1) if not above else range(edge + 1, edge + 7))


@pytest.mark.parametrize("spokes", [5, 6, 40])
def test_long_rows(cuda_ok, spokes):
    cfg = NetworkConfig(side=1.0, n_cnts=spokes + 1, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0))
    fast, r_fast, system = solve(fan_network(spokes, cfg), cfg, True)
    general, r_general, _ = solve(fan_network(spokes, cfg), cfg, False)
    assert abs(r_fast - r_general) <= 1e-9 * r_general
