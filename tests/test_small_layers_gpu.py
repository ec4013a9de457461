"""Batches of small layers, taken by the warp below 64 points: layer sizes around
32 and 64 points and the average size where the rule turns, exact ties and
duplicates, search boxes at the grid's edge, both input orders, ordered and
event-order batches.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu


def _batch(rng, events, layer_sizes, lattice, shuffled):
    counts = rng.choice(layer_sizes, (events, 100))
    off = np.concatenate([[0], np.cumsum(counts.sum(1))]).astype(np.int64)
    n = int(off[-1])
    layer = np.repeat(np.tile(np.arange(100), events), counts.ravel()).astype(np.int32)
    if lattice:  # exact distance and density ties, duplicated points, the grid's edge
        x = (rng.integers(-6, 7, n) * 0.5 - 248.0 * (layer % 3 == 0)).astype(np.float32)
        y = (rng.integers(-6, 7, n) * 0.5 + 248.0 * (layer % 5 == 0)).astype(np.float32)
        w = rng.integers(0, 3, n).astype(np.float32)
    else:
        x, y = (rng.normal(0, 4, n).astype(np.float32) for _ in range(2))
        w = rng.exponential(1.0, n).astype(np.float32)
    if shuffled:
        for e in range(events):
            p = off[e] + rng.permutation(off[e + 1] - off[e])
            for a in (x, y, layer, w):
                a[off[e]:off[e + 1]] = a[p]
    return off, x, y, layer, w


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("events,layer_sizes", [(2, (0, 1, 2)), (8, (31, 32, 33)), (8, (63, 64, 65)), (8, (0, 1, 63, 64, 150)),
                                                (8, (80,)), (8, (81,)), (420, (0, 1, 5))])
@pytest.mark.parametrize("prm", [(1.3, 2.0, 2.0), (7.0, 3.0, 1.5)])
def test_small_layers(cuda_lib, events, layer_sizes, lattice, shuffled, prm):
    rng = np.random.default_rng(events + layer_sizes[-1])
    off, x, y, layer, w = _batch(rng, events, layer_sizes, lattice, shuffled)
    algo = C.Clusterizer(*prm)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    assert_bitexact(got, oracle.clue2d_batch(off, x, y, layer, w, *prm, n_threads=4))


def test_small_layers_not_finite(cuda_lib):
    rng = np.random.default_rng(3)
    off, x, y, layer, w = _batch(rng, 8, (40, 63), False, False)
    n = x.size
    for a in (x, y, w):
        a[rng.integers(0, n, 200)] = np.nan
        a[rng.integers(0, n, 200)] = np.inf
        a[rng.integers(0, n, 200)] = -np.inf
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    want = oracle.clue2d_batch(off, x, y, layer, w, 1.3, 2.0, 2.0, n_threads=4)
    for k in ("nearestHigher", "isSeed", "clusterIndex"):
        assert np.array_equal(got[k], want[k]), k
    for k in ("rho", "delta"):  # a NaN matches any NaN
        same = (got[k].view(np.int32) == want[k].view(np.int32)) | (np.isnan(got[k]) & np.isnan(want[k]))
        assert same.all(), k
