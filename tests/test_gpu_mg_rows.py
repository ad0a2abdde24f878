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
