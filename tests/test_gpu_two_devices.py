"""Contexts and batches on two devices of one process: kernel attributes (shared memory above 48 KB,
16-CTA clusters) belong to a device and have to be set on each."""
import numpy as np
import pytest
from test_gpu_batch_clusters import system
from test_gpu_jacobi_sizes import ladder

from cicy_geom_b200 import batch as BT
from cicy_geom_b200.device import Context

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_devices(cuda_ok):
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")


@pytest.mark.parametrize("rungs,pre", [(60, 3), (700, 3), (700, 0), (700, 2)])
def test_networks(two_devices, rungs, pre):
    cfg, net = ladder(rungs)
    r = []
    for device in (0, 1):
        with Context(device) as ctx:
            ctx.set_solver(preconditioner=pre)
            ctx.upload(net)
            r.append(list(ctx.network_to_conductance(cfg.params()).resistances))
    assert r[0] == r[1]


def test_batches(two_devices):
    rng = np.random.default_rng(0)
    systems, x = [system(n, rng) for n in (700, 1500, 2500)], []
    for device in (0, 1):
        bs = BT.BatchSolver(systems, tol=1e-13, device=device)
        try:
            bs.enable_multigrid()
            bs.set_method(1)
            bs.solve()
            assert (bs.results()[2] == 1).all()
            x.append(bs.solutions())
        finally:
            bs.close()
    assert all(np.array_equal(a, b) for a, b in zip(*x))
