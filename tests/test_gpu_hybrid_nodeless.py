"""Junctions of a mixed network whose GNP point is in no GNP's point list: such a point has no node, the
system skips its junctions, and the backbone has to drop them without reading a voltage for them."""
import numpy as np
import pytest
from test_hybrid_electrical import _csr, hybrid_arrays, hybrid_state

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tag", ["s", "m"])
def test_unlisted_points(cuda_ok, tmp_path, tag):
    h, p, z, f = hybrid_state(tag, str(tmp_path))
    nclu = len(f["flow_family"])
    kept = _csr(z, f"e_c{nclu - 1}_bb_elements")
    # an end element of a CNT of the first cluster that the backbone does not keep
    cnt = next(c for c in h["clusters_cnt"][0] if h["elements"][c][-1] not in kept[c])
    gnps = h["clusters_gnp"][0]
    P = len(h["points_gnp"])
    h["points_gnp"] += [tuple(h["gnp_geom"][gnps[0]][1]), tuple(h["gnp_geom"][gnps[-1]][1])]
    h["junctions_gnp"].append((P, gnps[0], P + 1, gnps[-1], 0.001))
    h["cluster_gnp_junctions"][0].append(len(h["junctions_gnp"]) - 1)
    h["junctions_mixed"].append((h["elements"][cnt][-1], cnt, P, gnps[0], 0.001))
    h["cluster_mix_junctions"][0].append(len(h["junctions_mixed"]) - 1)
    prm = NetworkConfig(side=2.0, n_cnts=1, seed=0, tolerance=1e-10, vdw=0.00034, tunnel=0.0018).params()
    prm.resistances[0], prm.resistances[1], prm.resistances[2] = 1, 0, 0
    with Context(0) as ctx:
        ctx.upload(HostNetwork.from_arrays(h["net"]))
        r = ctx.hybrid_electrical(hybrid_arrays(h), prm, 1e-4, 1.0)
        for j in range(nclu):
            g, m = ctx.hybrid_junctions(j)
            assert g.tolist() == z[f"e_c{j}_bb_gnp_junctions"].tolist() and m.tolist() == z[f"e_c{j}_bb_mix_junctions"].tolist()
        bp, bi = ctx.elements(1)
        assert [list(bi[bp[c]:bp[c + 1]]) for c in range(len(bp) - 1)] == kept
    np.testing.assert_allclose(np.array(r.resistances), z["flow_resistances"], rtol=1e-6)  # the tolerance of the golden comparison
