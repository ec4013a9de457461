"""The bridge's eta and phi over many clusters of one point each, against the double
formulas.  The two-float forms hand over to the double form wherever its rounding
is in doubt, so each field is the double form's, bit for bit; a CPU's double
arc tangent and asinh differ from the GPU's by an ulp or two of a double, which
rounds to another float once in some 2^27 values: at most one such cluster is
allowed here, and by one ulp."""
import numpy as np
import pytest

import clue_gb300 as C
from clue_gb300 import synthetic as S
from oracle import bridge as OB

from _util import max_ulp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("place", ["ring", "near", "far", "steep", "lattice"])
def test_eta_and_phi(cuda_lib, place):
    import torch
    rng = np.random.default_rng(len(place))
    n = 200000
    r = {"ring": rng.uniform(20, 250, n), "near": 10.0 ** rng.uniform(-4, 1, n), "far": rng.uniform(250, 5000, n),
         "steep": rng.uniform(0.1, 250, n), "lattice": rng.uniform(1, 250, n)}[place]
    phi = rng.uniform(-np.pi, np.pi, n)
    if place == "steep":  # beside the axes and the diagonals, where the arc tangent's pieces meet
        phi = np.round(phi / (np.pi / 8)) * (np.pi / 8) + rng.normal(0, 1e-3, n)
    x, y = (r * np.cos(phi)).astype(np.float32), (r * np.sin(phi)).astype(np.float32)
    if place == "lattice":
        x, y = np.round(x * 4) / 4, np.round(y * 4) / 4
    w = np.ones(n, np.float32)
    lz = np.concatenate([S.layer_z(), -S.layer_z(), np.float32([0.5, 3, 40, 1e4, -7e5])]).astype(np.float32)
    layer = rng.integers(0, lz.size, n).astype(np.int32)
    ci, seed = np.arange(n, dtype=np.int32), np.ones(n, np.int32)
    off = np.array([0, n], np.int64)
    _, want = OB.layer_clusters(off, x, y, layer, w, seed, ci, lz)
    d = [torch.from_numpy(v).cuda() for v in (x, y, layer, w)]
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    _, got = algo.layer_clusters(off, *d, dict(isSeed=torch.from_numpy(seed).cuda(), clusterIndex=torch.from_numpy(ci).cuda()),
                                 layer_z=lz)
    got = {k: v.cpu().numpy() for k, v in got.items()}
    algo.close()
    for k in want:
        differ = np.count_nonzero(got[k].view(np.int32) != np.asarray(want[k]).view(np.int32))
        if k in ("eta", "phi"):
            assert differ <= 1 and max_ulp(got[k], want[k]) <= 1, (k, differ)
        else:
            assert differ == 0, (k, differ)
