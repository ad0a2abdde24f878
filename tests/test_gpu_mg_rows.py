"""Multigrid hierarchies with long coarse rows: the row gather deals rows by their
number of terms to a warp, a small CTA, a large CTA or a large CTA sorting in global
memory, so hubs just below and above each limit go through different kernels."""
import numpy as np
import pytest

from cicy_geom_b200 import batch as BT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 31, 511, 513, 2047, 2049, 8191, 8193])
def test_hub_rows_against_direct_solve(cuda_ok, degree):
    """A grounded ring of 9,000 one-node chains with three hubs of `degree` spokes each:
    eigenvalues lie in [1, 2 + 2 (4 + 3 degree)] and the solve stops at |r| <= 1e-13 |b|, so
    |x - x*| <= 1e-13 |b| with |b| <= sqrt(9000) max |b|: below 1e-10 for b of order 1."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sla

    n = 9000
    rng = np.random.default_rng(degree)
    i = np.arange(n)
    e = [np.stack([i, (i + 1) % n])]
    for hub in (17, 4000, 8999):
        spokes = rng.permutation(np.setdiff1d(i, [hub, (hub + 1) % n, (hub - 1) % n]))[: degree - 2]
        e.append(np.stack([np.full(len(spokes), hub), spokes]))
    e = np.concatenate(e, axis=1)
    W = sp.coo_matrix((rng.uniform(0.5, 2.0, e.shape[1]), (e[0], e[1])), shape=(n, n)).tocsr()
    W = W + W.T
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + 1.0) - W).tocsr()
    A.sort_indices()
    b = rng.uniform(-1.0, 1.0, n)
    bs = BT.BatchSolver([{"A": A, "b": b, "x0": np.zeros(n), "chain_start": i, "chain_len": np.ones(n, int)}], tol=1e-13)
    try:
        bs.enable_multigrid()
        bs.set_method(1)
        bs.solve()
        assert (bs.results()[2] == 1).all()
        x = bs.solutions()[0]
    finally:
        bs.close()
    assert np.max(np.abs(x - sla.spsolve(A.tocsc(), b))) < 1e-10


@pytest.mark.parametrize("spokes", [1400, 2200])
def test_grid_kernel_with_long_rows(cuda_ok, spokes):
    """A fan of CNTs on one end point through the grid kernel: coarse rows of hundreds of entries
    (a CTA's phase in several batches) and, with 2,200 spokes, one of more than a batch holds.
    Both preconditioners stop at 1e-13, as in the other comparisons of solvers."""
    from test_gpu_assembly import fan_network

    from cicy_geom_b200.device import Context
    from cicy_geom_b200.network import NetworkConfig

    cfg = NetworkConfig(side=1.0, n_cnts=spokes + 1, seed=0, tolerance=1e-13, tolerance_unit=1e-13, resistances=(1, 0, 0))
    net, r = fan_network(spokes, cfg), {}
    for pre in (0, 3):
        with Context(0) as ctx:
            ctx.set_solver(preconditioner=pre, cluster=False)
            ctx.upload(net)
            res = ctx.network_to_conductance(cfg.params())
            assert all(s.rel_residual <= 1e-10 for s in res.solves[:res.n_solves])
            r[pre], S = res.resistances[0], ctx.system(0)
    assert (np.diff(S["row_ptr"]) + np.bincount(S["col_ind"], minlength=len(S["diag"]))).max() >= spokes
    assert 0 < r[0] < 1e18 and abs(r[3] - r[0]) <= 1e-9 * r[0]
