"""Layers in HBM scratch, which keep their points' order in the searches: layer
sizes around the on-chip capacities, search boxes of one to many columns, both
input orders, a single event and a batch.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("prm", [(1.3, 2.0, 2.0), (3.0, 2.0, 2.0), (9.0, 20.0, 1.5)])
@pytest.mark.parametrize("sizes", [(4096, 4097), (15000, 300, 0, 1), (257,), (9000, 2000, 5000)])
@pytest.mark.parametrize("events", [1, 12])
def test_layers_over_the_capacity(cuda_lib, events, sizes, prm, shuffled):
    rng = np.random.default_rng(events + sizes[0])
    layer = np.concatenate([np.full(s, 7 * l + 1, np.int32) for l, s in enumerate(sizes)] * events)
    n = layer.size
    off = np.arange(events + 1, dtype=np.int64) * sum(sizes)
    x, y = (rng.uniform(-120, 120, n).astype(np.float32) for _ in range(2))
    w = rng.exponential(1.0, n).astype(np.float32)
    if shuffled:
        for e in range(events):
            layer[off[e]:off[e + 1]] = rng.permutation(layer[off[e]:off[e + 1]])
    algo = C.Clusterizer(*prm)
    algo.set_tuning(layer_capacity=256, big_capacity=2048)
    small = algo.run_batch(off, x, y, layer, w)
    algo.close()
    algo = C.Clusterizer(*prm)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    want = oracle.clue2d_batch(off, x, y, layer, w, *prm, n_threads=8)
    assert_bitexact(got, want)
    assert_bitexact(small, want)


@pytest.mark.parametrize("events", [1, 3, 12])
@pytest.mark.parametrize("n,rhoc", [(4200, 1.0), (20000, 1.0), (9000, 1e9)])
def test_long_chains(cuda_lib, events, n, rhoc):
    """Points on a line whose density rises along it: chains of thousands of steps,
    which end at a seed or at an outlier."""
    x = np.tile(np.linspace(-245, 245, n), events).astype(np.float32)
    y = np.zeros(n * events, np.float32)
    w = np.tile(np.linspace(1, 40, n), events).astype(np.float32)
    layer = np.full(n * events, 3, np.int32)
    off = np.arange(events + 1, dtype=np.int64) * n
    algo = C.Clusterizer(1.3, rhoc, 2.0)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    assert_bitexact(got, oracle.clue2d_batch(off, x, y, layer, w, 1.3, rhoc, 2.0, n_threads=8))
