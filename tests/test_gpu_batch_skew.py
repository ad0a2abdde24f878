"""Batched multigrid with one system much larger than the others, which keeps 16-CTA clusters whatever
the number of systems (csrc/batch_shape.h): every system against a direct solve, in the order given."""
import numpy as np
import pytest
import scipy.sparse.linalg as sla
from test_gpu_batch_clusters import system

from cicy_geom_b200 import batch as BT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [8, 40])
def test_one_large_system(cuda_ok, count):
    rng = np.random.default_rng(count)
    systems = [system(int(n), rng) for n in rng.integers(200, 900, count)]
    systems.insert(count // 2, system(60_000, rng))
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
