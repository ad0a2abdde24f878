"""The explicit inverses of the chain blocks: on a matrix of uncoupled chains they are the exact
inverse, so preconditioned CG is done after one iteration (a second for rounding)."""
import numpy as np
import pytest
import scipy.sparse as sp

from cicy_geom_b200 import batch as BT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[1], [2], [31], [32], [1, 32, 2, 31, 16, 17], list(range(1, 33)) * 40])
def test_exact_on_uncoupled_chains(cuda_ok, lengths):
    rng = np.random.default_rng(len(lengths))
    n, start = sum(lengths), np.concatenate([[0], np.cumsum(lengths)[:-1]])
    g = 10.0 ** rng.uniform(-1, 1, n)  # coupling of row i to i + 1, none across chains
    g[start + np.array(lengths) - 1] = 0
    left = np.concatenate([[0], g[:-1]])
    A = sp.diags([left + g + 0.5, -g[:-1], -g[:-1]], [0, 1, -1]).tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    x = rng.uniform(-1, 1, n)
    bs = BT.BatchSolver([{"A": A, "b": A @ x, "x0": np.zeros(n), "chain_start": start, "chain_len": np.array(lengths)}], tol=1e-10)
    try:
        bs.set_method(2)
        bs.solve()
        iterations, rel, flags = bs.results()
        got = bs.solutions()[0]
    finally:
        bs.close()
    assert flags[0] == 1 and iterations[0] <= 2
    # |A^-1| <= 2 (rows sum to 0.5), so |x - x*| <= 2 |r| <= 2e-10 |b|, |b| <= sqrt(n) 41
    assert np.max(np.abs(got - x)) <= 2e-10 * 41 * np.sqrt(n)
