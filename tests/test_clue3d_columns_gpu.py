"""CLUE3D rows that hold several entries in few phi columns, as many as a search
window spans and more, from two entries to hundreds, at the window's ends and
across the phi wrap; within and beyond the staged columns.  Bit-exact against the
oracle."""
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


@pytest.mark.parametrize("siblings", [1, 3])
@pytest.mark.parametrize("columns", [1, 2, 7])
@pytest.mark.parametrize("first", [0, 62, 124])
@pytest.mark.parametrize("n,etas", [(400, 0.02), (3000, 0.02), (3000, 1.5), (9000, 0.3)])
def test_crowded_columns(cuda_lib, n, etas, first, columns, siblings):
    ev = S.clue3d_event(n + first, n_clusters=n, n_layers=30, eta_range=(1.5, 1.5 + etas))
    rng = np.random.default_rng(columns)
    phi = (first + rng.uniform(0, columns, n)) % 126 * (2 * math.pi / 126) - math.pi
    ev["phi"] = phi.astype(np.float32)
    prm = dict(n_layers=30, density_sibling_layers=siblings, nh_sibling_layers=siblings)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out, nts = algo.run_clue3d(np.array([0, n], np.int64), ev, params=prm)
    algo.close()
    want, nt = oracle.clue3d(ev, **prm)
    assert int(nts[0]) == nt
    assert_bitexact({NAMES[k]: v for k, v in out.items()}, want, keys=tuple(NAMES.values()))
