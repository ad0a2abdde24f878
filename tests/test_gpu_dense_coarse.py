"""Dense coarsest levels around the sizes where the grid Gauss-Jordan's tile grows: ladders whose
chains (a rung each, the spines in blocks of 32 nodes) are the coarsest level.  The multigrid solve
agrees with Jacobi-PCG, and its unit pass stays at a two-level method's iterations (a wrong inverse
would cost hundreds; the real pass restarts at the rounding floor of this tolerance, so its count
says nothing)."""
import pytest
from test_gpu_jacobi_sizes import ladder

from cicy_geom_b200.device import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rungs", [n * 32 // 34 + d for n in (140, 384, 768, 960, 1152) for d in (-1, 0, 1)] + [1203])
def test_ladder_multigrid(cuda_ok, rungs):
    cfg, net = ladder(rungs)
    r, solves = {}, {}
    for pre in (0, 3):
        with Context(0) as ctx:
            ctx.set_solver(preconditioner=pre, cluster=False)
            ctx.upload(net)
            res = ctx.network_to_conductance(cfg.params())
            r[pre], solves[pre] = res.resistances[0], [(s.nodes, s.iterations, s.rel_residual) for s in res.solves[:res.n_solves]]
    assert [s[0] for s in solves[0]] == [s[0] for s in solves[3]]
    assert all(s[2] <= 1e-10 for s in solves[0] + solves[3]) and solves[3][0][1] <= 150
    assert 0 < r[0] < 1e18 and abs(r[3] - r[0]) <= 1e-9 * r[0]


@pytest.mark.parametrize("rungs", [70, 74, 75, 80])
def test_around_the_one_cluster_limit(cuda_ok, rungs):
    """Unit passes of 422 to 482 rows: the one-cluster kernel up to 450, the grid kernel above."""
    cfg, net = ladder(rungs)
    r = {}
    for pre, cluster in ((0, False), (3, True), (3, False)):
        with Context(0) as ctx:
            ctx.set_solver(preconditioner=pre, cluster=cluster)
            ctx.upload(net)
            res = ctx.network_to_conductance(cfg.params())
            assert all(s.rel_residual <= 1e-10 for s in res.solves[:res.n_solves])
            assert pre == 0 or res.solves[0].kernel == 2
            r[pre, cluster] = res.resistances[0]
    for k in ((3, True), (3, False)):
        assert 0 < r[0, False] < 1e18 and abs(r[k] - r[0, False]) <= 1e-9 * r[0, False]
