"""Contacts, junctions, labels and clusters of networks whose CNTs have few, many (above one warp's
128) and very many (above one CTA's 2,048) contacts, of points far outside the window, of two
percolated clusters, and of more CNTs than the quadratic label ranking takes.  All bit-exact."""
import numpy as np
import pytest

from cicy_geom_b200.device import Context
from cicy_geom_b200.network import HostNetwork, NetworkConfig
from oracle import cicy_oracle as O

pytestmark = pytest.mark.gpu


def spines(crossings, n_spines, specks, window, seed):
    """Spines along x, `crossings` short CNTs across each, `specks` two-point CNTs (half of them in touching pairs)."""
    rng = np.random.default_rng(seed)
    lines = []
    for s in range(n_spines):
        y = 0.25 + 0.5 * s / max(n_spines - 1, 1)
        lines.append(np.stack([np.linspace(0, 1, 401), np.full(401, y), np.full(401, 0.5)], 1))
    for s in range(n_spines):
        y = 0.25 + 0.5 * s / max(n_spines - 1, 1)
        for _ in range(crossings):
            c = np.array([rng.uniform(0.02, 0.98), y, 0.5])
            u = rng.normal(size=3)
            u[0] = 0
            u /= np.linalg.norm(u)
            lines.append(c + np.linspace(-0.02, 0.02, 9)[:, None] * u)
    c = rng.uniform(0.05, 0.95, size=(specks, 3))
    c[1::2] = c[::2] + [0.0108, 0, 0]
    lines += [np.stack([p, p + [0, 0.004, 0.001]]) for p in c]
    xyz, ptr, n = np.concatenate(lines), np.concatenate([[0], np.cumsum([len(v) for v in lines])]), len(lines)
    faces = [[], [], list(range(n_spines)), [], list(range(n_spines)), []]
    pts = [[], [], [int(ptr[i]) for i in range(n_spines)], [], [int(ptr[i + 1]) - 1 for i in range(n_spines)], []]
    off = lambda v: np.concatenate([[0], np.cumsum([len(x) for x in v])])
    return {"x": xyz[:, 0], "y": xyz[:, 1], "z": xyz[:, 2], "flag": np.repeat(np.arange(n), np.diff(ptr)), "structure_ptr": ptr,
            "structure_idx": np.arange(len(xyz)), "radii": np.full(n, 0.005), "cnts_inside": rng.permutation(n),
            "boundary_cnt_ptr": off(faces), "boundary_cnt_idx": sum(faces, []), "boundary_pts_ptr": off(pts),
            "boundary_pts_idx": sum(pts, []), "window": window}


UNIT = [0, 0, 0, 1, 1, 1, 1, 1, 1]


@pytest.mark.parametrize("crossings,n_spines,specks,window,contacts", [
    (0, 1, 2, UNIT, 0), (20, 1, 0, UNIT, 20), (200, 2, 40, UNIT, 129), (1500, 1, 0, UNIT, 2049), (1500, 2, 0, UNIT, 2049),
    (150, 2, 100, [0.4, 0.2, 0.45, 0.1, 0.1, 0.1, 0.5, 0.3, 0.55], 129), (3, 9, 0, UNIT, 0), (10, 1, 60_010, UNIT, 0)])
def test_contacts_against_oracle(cuda_ok, crossings, n_spines, specks, window, contacts):
    a = spines(crossings, n_spines, specks, window, seed=crossings + specks)
    cfg = NetworkConfig(side=1.0, n_cnts=len(a["radii"]), seed=0)
    with Context(0) as ctx:
        ctx.upload(HostNetwork.from_arrays(a))
        p = cfg.params()
        ctx.contact_grid(p)
        ctx.clusters(p)
        pa, cb, pb, d = ctx.point_contacts()
        lab, nl = ctx.labels()
        junc = ctx.junctions()
        ep, ei = ctx.elements(0)
        cl = ctx.percolated_clusters(0)
    a = {k: np.asarray(v) for k, v in a.items()}
    op = O.params_from_config(cfg)
    labels, n_labels, pc, ce = O.label_cnts(a, op, O.contact_grid(a, op)[2])
    junctions, elements = O.compress_junctions(a, op, pc, ce)
    clusters, families, cj = O.percolation(a, labels, n_labels, junctions)
    assert np.bincount(a["flag"][pa], minlength=1).max(initial=0) >= contacts
    keys = sorted(pc)
    assert list(zip(pa, cb)) == keys and list(pb) == [pc[k][0] for k in keys] and list(d) == [pc[k][1] for k in keys]
    assert nl == n_labels and np.array_equal(lab, labels)
    assert list(zip(*junc)) == junctions
    assert {i: list(ei[ep[i]:ep[i + 1]]) for i in range(len(lab)) if ep[i + 1] > ep[i]} == elements
    cut = lambda ptr, idx: [list(idx[ptr[i]:ptr[i + 1]]) for i in range(len(ptr) - 1)]
    assert list(cl["family"]) == families and cut(cl["ptr"], cl["idx"]) == clusters and cut(cl["junc_ptr"], cl["junc_idx"]) == cj
