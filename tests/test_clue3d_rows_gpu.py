"""CLUE3D rows at the limits of the staged searches: columns held twice in more
rows of a slab than it has second-entry slots, columns held three times and
more (rows walked entry by entry), and phi on the edges of the 32-column words
and of the wrap.  Bit-exact against the oracle."""
import math

import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

NAMES = dict(rho="rho", delta_transverse="delta_t", delta_layers="delta_l", nh_layer="nh_layer", nh_index="nh_idx",
             isSeed="isSeed", tracksterIndex="tracksterIndex")


def _event(kind):
    ev = S.clue3d_event(5, n_clusters=6000, n_layers=94)
    rng = np.random.default_rng(9)
    if kind == "pairs":  # every second cluster beside the one before it: nearly every row repeats a column
        for k in ("eta", "phi", "layer", "z", "r_over_absz"):
            ev[k][1::2] = ev[k][0::2]
    elif kind == "triples":  # a narrow phi band: three entries and more in most columns
        ev["phi"] = rng.uniform(-0.3, 0.3, ev["phi"].size).astype(np.float32)
    else:  # a few ulps around every bin edge that starts a word, and around the wrap
        edges = np.array([32, 64, 96, 124, 125, 126, 0, 1, 2], np.float64) * (2 * math.pi / 126) - math.pi
        phi = rng.choice(edges, ev["phi"].size).astype(np.float32)
        phi = (phi + rng.integers(-3, 4, phi.size).astype(np.float32) * np.float32(2.4e-7)).astype(np.float32)
        ev["phi"] = np.clip(phi, -np.float32(math.pi), np.float32(math.pi))
    return ev


@pytest.mark.parametrize("siblings", [2, 3])
@pytest.mark.parametrize("kind", ["pairs", "triples", "edges"])
def test_rows(cuda_lib, kind, siblings):
    ev = _event(kind)
    prm = dict(n_layers=94, density_sibling_layers=siblings, nh_sibling_layers=siblings)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out, nts = algo.run_clue3d(np.array([0, ev["z"].size], np.int64), ev, params=prm)
    algo.close()
    want, nt = oracle.clue3d(ev, **prm)
    assert int(nts[0]) == nt
    assert_bitexact({NAMES[k]: v for k, v in out.items()}, want, keys=tuple(NAMES.values()), label=kind)


@pytest.mark.parametrize("siblings", [2, 3])
@pytest.mark.parametrize("kind,n", [("row", 6000), ("row", 16000), ("column", 6000), ("column", 2000),
                                    ("wide", 60000), ("row", 40000)])
def test_crowded_rows(cuda_lib, kind, n, siblings):
    """Rows searched by their entries' columns, within the room that a slab has
    for staged columns and beyond it: every cluster of a layer in its first eta row
    (16,000 clusters: more columns than fit), or in one phi column (more such rows
    than fit), some of them at the wrap; and events whose slabs are searched in
    global memory, where most rows repeat a column."""
    ev = S.clue3d_event(11, n_clusters=n, n_layers=94)
    rng = np.random.default_rng(n)
    if kind == "row":
        ev["eta"] = np.minimum(ev["eta"], np.float32(1.4999))
    elif kind == "column":
        ev["phi"] = rng.uniform(3.12, math.pi, n).astype(np.float32) * rng.choice([-1, 1], n).astype(np.float32)
    prm = dict(n_layers=94, density_sibling_layers=siblings, nh_sibling_layers=siblings)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out, nts = algo.run_clue3d(np.array([0, n], np.int64), ev, params=prm)
    algo.close()
    want, nt = oracle.clue3d(ev, **prm)
    assert int(nts[0]) == nt
    assert_bitexact({NAMES[k]: v for k, v in out.items()}, want, keys=tuple(NAMES.values()), label=kind)


@pytest.mark.parametrize("layers,siblings,n", [(94, 2, 21056), (94, 2, 21057), (94, 3, 19000), (94, 3, 33000), (10, 2, 3000),
                                               (7, 3, 1500), (1, 2, 700)])
def test_slabs_in_parts(cuda_lib, layers, siblings, n):
    """Slabs around the size from which they may be searched in halves or single
    layers, with an event beyond it and a crowded layer beside small ones, and layer
    counts that leave a slab of one to three layers."""
    rng = np.random.default_rng(n + layers)
    evs = [S.clue3d_event(21, n_clusters=n, n_layers=max(layers, 2)), S.clue3d_event(22, n_clusters=900, n_layers=max(layers, 2))]
    for ev in evs:
        ev["layer"] = np.minimum(ev["layer"], layers - 1).astype(np.int32)
    crowd = rng.random(n) < 0.1
    evs[0]["layer"][crowd] = layers // 2
    off = np.array([0, n, n + 900], np.int64)
    both = {k: np.concatenate([ev[k] for ev in evs]) for k in evs[0]}
    prm = dict(n_layers=layers, density_sibling_layers=siblings, nh_sibling_layers=siblings)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out, nts = algo.run_clue3d(off, both, params=prm)
    algo.close()
    for e, ev in enumerate(evs):
        want, nt = oracle.clue3d(ev, **prm)
        assert int(nts[e]) == nt
        assert_bitexact({NAMES[k]: v[off[e]:off[e + 1]] for k, v in out.items()}, want, keys=tuple(NAMES.values()),
                        label=f"event {e}")
