"""Batches of mostly small layers, taken by the warp below 64 points, beside some
above the first pass's capacity, in the sizes whose passes run side by side when
captured, in turn, or in event order: three runs each (direct, captured,
replayed), both input orders.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)
KEYS = ("rho", "delta", "nearestHigher", "isSeed", "clusterIndex")


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("events", [5, 10, 40, 300, 420])
def test_both_kinds(cuda_lib, events, shuffled):
    import torch
    rng = np.random.default_rng(events)
    counts = rng.choice([0, 1, 20, 63, 64], (events, 100))
    large = rng.random(counts.shape) < 0.007
    counts[large] = rng.integers(1400, 5000, int(large.sum()))
    counts[0, 5] = 5000  # above both capacities
    off = np.concatenate([[0], np.cumsum(counts.sum(1))]).astype(np.int64)
    n = int(off[-1])
    assert n <= 80 * 100 * events
    layer = np.repeat(np.tile(np.arange(100), events), counts.ravel()).astype(np.int32)
    size = np.repeat(counts.ravel(), counts.ravel())
    side = np.where(size > 64, 100, 8)
    x, y = ((rng.uniform(-1, 1, n) * side).astype(np.float32) for _ in range(2))
    w = rng.exponential(1.0, n).astype(np.float32)
    if shuffled:
        for e in range(events):
            p = off[e] + rng.permutation(off[e + 1] - off[e])
            for a in (x, y, layer, w):
                a[off[e]:off[e + 1]] = a[p]
    want = oracle.clue2d_batch(off, x, y, layer, w, *PRM, n_threads=8)
    dev = [torch.from_numpy(v).cuda() for v in (x, y, layer, w)]
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    algo = C.Clusterizer(*PRM)
    for _ in range(3):
        for v in out.values():
            v.zero_()
        torch.cuda.synchronize()
        algo.run_batch(off, *dev, out=out, flags=C.DEVICE_MEMORY)
        algo.synchronize()
        assert_bitexact({k: v.cpu().numpy() for k, v in out.items()}, want)
    algo.close()
