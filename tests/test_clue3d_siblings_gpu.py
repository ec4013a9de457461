"""CLUE3D with wide sibling windows, whose rows fit the searches' staging area
for half a slab, for a single layer, or not at all, and mixed widths of the two
searches, with sparse and crowded layers.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

NAMES = dict(rho="rho", delta_transverse="delta_t", delta_layers="delta_l", nh_layer="nh_layer", nh_index="nh_idx",
             isSeed="isSeed", tracksterIndex="tracksterIndex")


@pytest.mark.parametrize("layers", [94, 13, 11, 3])
@pytest.mark.parametrize("density,nearest", [(4, 4), (5, 5), (6, 6), (9, 2), (3, 7), (100, 100), (-1, 4)])
@pytest.mark.parametrize("n", [1500, 12000])
def test_wide_windows(cuda_lib, layers, density, nearest, n):
    evs = [S.clue3d_event(41, n_clusters=n, n_layers=layers), S.clue3d_event(42, n_clusters=300, n_layers=layers)]
    evs[0]["layer"][::5] = layers // 2
    off = np.array([0, n, n + 300], np.int64)
    both = {k: np.concatenate([ev[k] for ev in evs]) for k in evs[0]}
    prm = dict(n_layers=layers, density_sibling_layers=density, nh_sibling_layers=nearest)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out, nts = algo.run_clue3d(off, both, params=prm)
    algo.close()
    for e, ev in enumerate(evs):
        want, nt = oracle.clue3d(ev, **prm)
        assert int(nts[e]) == nt
        assert_bitexact({NAMES[k]: v[off[e]:off[e + 1]] for k, v in out.items()}, want, keys=tuple(NAMES.values()),
                        label=f"event {e}")
