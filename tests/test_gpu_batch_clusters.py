"""Batched multigrid with more systems than 16-CTA clusters fit at once (8-CTA clusters), and more
than two rounds of those (4-CTA): every system against a direct solve, in the order given."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from cicy_geom_b200 import batch as BT

pytestmark = pytest.mark.gpu


def system(n, rng):
    """A grounded ring of n rows in chains of up to seven: eigenvalues in [1, 1 + 2 * 6]."""
    i = np.arange(n)
    e = np.concatenate([np.stack([i, (i + 1) % n]), np.stack([i, (i + n // 3) % n])], axis=1)
    W = sp.coo_matrix((rng.uniform(0.5, 1.5, e.shape[1]), (e[0], e[1])), shape=(n, n)).tocsr()
    W = W + W.T
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + 1.0) - W).tocsr()
    A.sort_indices()
    start = np.arange(0, n, 7)
    return {"A": A, "b": rng.uniform(-1, 1, n), "x0": np.zeros(n), "chain_start": start, "chain_len": np.minimum(7, n - start)}


@pytest.mark.parametrize("count", [3, 9, 40, 75])
def test_uneven_systems(cuda_ok, count):
    rng = np.random.default_rng(count)
    systems = [system(int(n), rng) for n in rng.integers(60, 3000, count)]
    bs = BT.BatchSolver(systems, tol=1e-13)
    try:
        bs.enable_multigrid()
        bs.set_method(1)
        bs.solve()
        flags, x = bs.results()[2], bs.solutions()
    finally:
        bs.close()
    assert (flags == 1).all()
    for s, got in zip(systems, x):  # |x - x*| <= |r| <= 1e-13 |b| (smallest eigenvalue 1)
        assert np.max(np.abs(got - sla.spsolve(s["A"].tocsc(), s["b"]))) < 1e-10
