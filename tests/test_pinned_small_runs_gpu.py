"""Small host-memory runs from page-locked arrays, alone and mixed with pageable
ones, on both sides of the size up to which they are staged (448 KB in all: 12,743
points, 7,645 layer clusters), on the handle's stream and a caller's.  Bit-exact
against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)
NAMES = dict(rho="rho", delta_transverse="delta_t", delta_layers="delta_l", nh_layer="nh_layer", nh_index="nh_idx",
             isSeed="isSeed", tracksterIndex="tracksterIndex")


def _host(a, pinned):
    import torch
    return torch.from_numpy(np.array(a)).pin_memory().numpy() if pinned else np.array(a)


@pytest.mark.parametrize("caller", [False, True])
@pytest.mark.parametrize("kind", ["pinned", "pageable layer", "pageable outputs"])
@pytest.mark.parametrize("n", [12743, 12744, 32768, 32769])
def test_clue2d(cuda_lib, n, kind, caller):
    import torch
    rng = np.random.default_rng(n)
    ev = dict(x=rng.normal(0, 40, n).astype(np.float32), y=rng.normal(0, 40, n).astype(np.float32),
              layer=rng.integers(0, 100, n).astype(np.int32), weight=rng.exponential(1.0, n).astype(np.float32))
    host = {k: _host(v, kind != "pageable layer" or k != "layer") for k, v in ev.items()}
    out = {k: _host(v, kind != "pageable outputs") for k, v in C.empty_outputs(n).items()}
    stream = torch.cuda.Stream() if caller else None
    algo = C.Clusterizer(*PRM, stream=stream.cuda_stream if caller else None)
    want = oracle.clue2d(*[ev[k] for k in ("x", "y", "layer", "weight")], *PRM)
    for _ in range(3):
        algo.run_batch(np.array([0, n], np.int64), *[host[k] for k in ("x", "y", "layer", "weight")], out=out)
        assert_bitexact(out, want)
    algo.close()


@pytest.mark.parametrize("n", [7645, 7646, 32769])
@pytest.mark.parametrize("pinned", [False, True])
def test_clue3d(cuda_lib, n, pinned):
    ev = S.clue3d_event(n, n_clusters=n, n_layers=94)
    host = {k: _host(v, pinned) for k, v in ev.items()}
    out = {k: _host(np.zeros(n, np.float32 if k in ("rho", "delta_transverse") else np.int32), pinned) for k in NAMES}
    algo = C.Clusterizer(*PRM)
    want, nt = oracle.clue3d(ev)
    for _ in range(2):
        got, nts = algo.run_clue3d(np.array([0, n], np.int64), host, out=out)
        assert int(nts[0]) == nt
        assert_bitexact({NAMES[k]: v for k, v in got.items()}, want, keys=tuple(NAMES.values()))
    algo.close()
