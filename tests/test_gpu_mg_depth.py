"""Multigrid hierarchies of the largest depth (16 levels).  A ladder whose rungs are lines of short
CNTs joined end to end, with equal couplings along a line: the matching then starts at the line's
ends only and takes a few rows off each line, so a level keeps 0.83-0.9 of the rows above it.  The
grid kernel records one shared-memory copy per operator set of every level, most of them here.  Line
lengths follow an exponential distribution; mean 26 ends in a dense coarsest level, mean 30 in one
that is too large for it."""
import numpy as np
import pytest

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig
from oracle import cicy_oracle as O

pytestmark = pytest.mark.gpu

LAYERS, LINES, POINTS = 8, 50, 450  # ladders above one another, rungs of each, points of a rung


def exponential(mean):
    n = LAYERS * LINES
    quantile = np.random.default_rng(0).permutation(-mean * np.log(1 - (np.arange(n) + 0.5) / n))
    return np.clip(np.round(quantile), 1, POINTS // 3).astype(int).reshape(LAYERS, LINES)


def lines_network(counts):
    """Short ladders (every rung then carries a current the backbone keeps), one CNT across them all;
    counts[layer, rung]: CNTs of each rung."""
    length = 4.9
    cfg = NetworkConfig(side=length, n_cnts=1, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0), gs_min=length / 60)
    y = 0.25 + np.arange(POINTS) / 100
    cnts = []
    for layer in range(len(counts)):
        for yy, lo, hi in ((y[0], -0.04, 1.6), (y[-1], 0.05, length + 0.04)):
            x = np.arange(round(lo * 100), round(hi * 100) + 1) / 100
            cnts.append(np.stack([x, np.full(len(x), yy), np.full(len(x), 0.5 + 0.1 * layer)], 1))
    z = 0.5 + np.arange(10 * (len(counts) - 1) + 1) / 100
    cnts.append(np.stack([np.full(len(z), 1.5), np.full(len(z), y[0] - 0.0108), z], 1))
    for k, count in enumerate(np.ravel(counts)):
        layer, rung = divmod(k, len(counts[0]))
        cnts += np.array_split(np.stack([np.full(POINTS, 0.06 + 0.02 * rung), y, np.full(POINTS, 0.5108 + 0.1 * layer + 1e-5 * (k % 7))], 1), count)
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cnts])])
    xyz, n = np.concatenate(cnts), len(cnts)
    return cfg, HostNetwork.from_arrays({
        "x": xyz[:, 0], "y": xyz[:, 1], "z": xyz[:, 2], "flag": np.repeat(np.arange(n), np.diff(ptr)), "structure_ptr": ptr,
        "structure_idx": np.arange(len(xyz)), "radii": np.full(n, cfg.radius), "window": [0, 0, 0] + 6 * [length]}).extract_window(cfg)


@pytest.mark.parametrize("mean", [26, 30])
def test_sixteen_levels(cuda_ok, mean):
    """Both passes (21,600 and 24,700 rows) against a direct solve: |x - x*| <= |b - A x| / lambda, for
    each of the two solutions compared, with lambda the smallest eigenvalue."""
    import scipy.sparse.linalg as sla

    cfg, net = lines_network(exponential(mean))
    with Context(0) as ctx:
        ctx.set_solver(preconditioner=3, smoothed=False)
        ctx.upload(net)
        res = ctx.network_to_conductance(cfg.params())
        systems = [ctx.system(i) for i in range(res.n_solves)]
    assert len(systems) == 2
    for s, S in zip(res.solves, systems):
        assert s.kernel == 2 and s.levels == 16 and s.rel_residual <= 1e-10
        A, b = O.full_matrix(S).tocsc(), S["b"]
        x, direct = S["voltages"][S["reserved"]:], sla.spsolve(A, b)
        lam = sla.eigsh(A, k=1, sigma=0, return_eigenvectors=False)[0]
        assert lam > 0 and np.linalg.norm(x - direct) <= (np.linalg.norm(b - A @ x) + np.linalg.norm(b - A @ direct)) / lam


@pytest.mark.parametrize("cnts,cluster,one_cluster", [(21, True, True), (21, False, False), (22, True, False), (22, False, False)])
def test_kernel_at_the_one_cluster_limit(cuda_ok, cnts, cluster, one_cluster):
    """Unit passes of 448 and 468 rows with more than 200 chains: the one-cluster kernel, up to 450 rows, has
    a dense coarsest level of at most 128 rows and so more levels; the grid kernel inverts level 1."""
    cfg, net = lines_network(np.full((2, 5), cnts))
    with Context(0) as ctx:
        ctx.set_solver(preconditioner=3, cluster=cluster)
        ctx.upload(net)
        s = ctx.network_to_conductance(cfg.params()).solves[0]
    assert s.nodes - s.reserved == 20 * cnts + 28 and s.kernel == 2 and s.rel_residual <= 1e-10
    assert s.levels > 2 if one_cluster else s.levels == 2
