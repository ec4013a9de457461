"""CLUE3D clusters whose phi reduces to bin 126 (-3 pi and 5 pi as floats): they
fall into the next eta row, and in a layer's last one into the next layer's first
row or, on the last layer, into a row behind all layers, which is searched as
the others are.  Outputs hold a pattern beforehand, so that a cluster left out
shows.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

NAMES = dict(rho="rho", delta_transverse="delta_t", delta_layers="delta_l", nh_layer="nh_layer", nh_index="nh_idx",
             isSeed="isSeed", tracksterIndex="tracksterIndex")
BIN_126 = np.array([-9.42477798461914, 15.707963943481445], np.float32)


def _event(n, layers, share, seed):
    ev = S.clue3d_event(seed, n_clusters=n, n_layers=max(layers, 2))
    rng = np.random.default_rng(seed)
    ev["layer"] = np.minimum(ev["layer"], layers - 1).astype(np.int32)
    at = rng.random(n) < share
    k = int(at.sum())
    ev["phi"][at] = rng.choice(BIN_126, k)
    ev["eta"][at] = rng.uniform(3.1, 3.3, k).astype(np.float32) * rng.choice([-1, 1], k).astype(np.float32)
    ev["layer"][at] = rng.integers(max(layers - 3, 0), layers, k)
    ev["r_over_absz"] = (1.0 / np.sinh(np.abs(ev["eta"]).astype(np.float64))).astype(np.float32)
    return ev


def test_phi_of_bin_126():
    o2pi, twopi = np.float32(1 / (2 * np.pi)), np.float32(2 * np.pi)
    norm = BIN_126 - np.round(BIN_126 * o2pi).astype(np.float32) * twopi
    assert ((norm.astype(np.float64) + np.pi) * np.float64(np.float32(126 / (2 * np.pi))) >= 126).all()


@pytest.mark.gpu
@pytest.mark.parametrize("layers,siblings,n,share", [(94, 3, 4000, 0.05), (94, 3, 40000, 0.02), (4, 2, 300, 0.3), (5, 2, 300, 0.3),
                                                     (1, 2, 200, 0.5), (8, 4, 900, 0.2), (94, 3, 1, 1.0)])
def test_row_behind_the_last_layer(cuda_lib, layers, siblings, n, share):
    evs = [_event(n, layers, share, 31), _event(500, layers, share, 32)]
    off = np.array([0, n, n + 500], np.int64)
    both = {k: np.concatenate([ev[k] for ev in evs]) for k in evs[0]}
    prm = dict(n_layers=layers, density_sibling_layers=siblings, nh_sibling_layers=siblings)
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    out = {k: np.full(n + 500, 12345, np.float32 if k in ("rho", "delta_transverse") else np.int32) for k in NAMES}
    out, nts = algo.run_clue3d(off, both, params=prm, out=out)
    algo.close()
    for e, ev in enumerate(evs):
        want, nt = oracle.clue3d(ev, **prm)
        assert_bitexact({NAMES[k]: v[off[e]:off[e + 1]] for k, v in out.items()}, want, keys=tuple(NAMES.values()),
                        label=f"event {e}")
        assert int(nts[e]) == nt
