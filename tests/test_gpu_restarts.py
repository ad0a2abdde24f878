"""Residual replacements sum r.r twice in a row; every CTA has to read all of the first sum's partials
before they are written again.  All sums of the solvers run in a fixed order, so a solve that restarts
gives the same iterations and the same voltages to the last bit each time."""
import numpy as np
import pytest
from test_gpu_jacobi_sizes import ladder

from cicy_geom_b200.device import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rungs,pre,cluster", [(2100, 0, False), (500, 2, False), (60, 3, True), (60, 3, False), (700, 3, False), (2100, 3, True)])
def test_restarted_solves_repeat(cuda_ok, rungs, pre, cluster):
    cfg, net = ladder(rungs)
    runs = []
    for _ in range(4):
        with Context(0) as ctx:
            ctx.set_solver(preconditioner=pre, cluster=cluster)
            ctx.upload(net)
            res = ctx.network_to_conductance(cfg.params())
            runs.append([(s.iterations, s.restarts, s.kernel, ctx.system(i)["voltages"]) for i, s in enumerate(res.solves[:res.n_solves])])
    assert sum(s[1] for s in runs[0]) > 0 and all(s[2] == (2 if pre == 3 else 0) for s in runs[0])
    for other in runs[1:]:
        assert [s[:3] for s in other] == [s[:3] for s in runs[0]]
        assert all(np.array_equal(s[3], t[3]) for s, t in zip(other, runs[0]))
