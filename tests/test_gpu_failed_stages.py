"""A stage that fails part of the way leaves its arrays half written: the calls after it that would read
them are refused (CICY_E_STATE), and a new network works in the same context."""
import pytest

from cicy_geom_b200 import _abi
from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig, generate_cnt_network

pytestmark = pytest.mark.gpu
INPUT, CAPACITY, STATE = 1, 2, 6
CFG = NetworkConfig(side=1.6, n_cnts=500, seed=3)


def refused(call, status):
    with pytest.raises(_abi.CicyError) as e:
        call()
    assert e.value.status == status


def check_usable(ctx, expected):
    refused(lambda: ctx.network_to_conductance(CFG.params()), STATE)
    ctx.generate_network(CFG)
    assert list(ctx.network_to_conductance(CFG.params()).resistances) == expected


@pytest.fixture
def ctx(cuda_ok):
    with Context(0) as c:
        c.generate_network(CFG)
        yield c


def test_generator_with_too_many_points(ctx):
    expected = list(ctx.network_to_conductance(CFG.params()).resistances)
    refused(lambda: ctx.generate_network(NetworkConfig(side=1.6, n_cnts=60_000, seed=1, step=1e-5)), CAPACITY)  # about 6e9
    check_usable(ctx, expected)


def test_upload_of_a_broken_structure(ctx):
    expected = list(ctx.network_to_conductance(CFG.params()).resistances)
    a = generate_cnt_network(NetworkConfig(side=1.6, n_cnts=900, seed=2)).extract_window(CFG).arrays()
    a["structure_idx"] = a["structure_idx"].copy()
    a["structure_idx"][[1, 2]] = a["structure_idx"][[2, 1]]
    refused(lambda: ctx.upload(HostNetwork.from_arrays(a)), INPUT)
    check_usable(ctx, expected)


def test_trim_of_another_layout(ctx):
    expected = list(ctx.network_to_conductance(CFG.params()).resistances)
    refused(lambda: ctx.extract_window(CFG), INPUT)  # the window has been trimmed already: runs and flags have gaps
    check_usable(ctx, expected)


def test_grid_with_too_many_points_in_a_region(ctx):
    p, one = CFG.params(), CFG.params()
    expected = list(ctx.network_to_conductance(p).resistances)
    one.gs_min[:] = [1.6] * 3  # one region of all points
    refused(lambda: ctx.contact_grid(one), CAPACITY)
    refused(lambda: ctx.clusters(p), STATE)
    assert list(ctx.network_to_conductance(p).resistances) == expected
