"""Seed numbering over events of many chunks: on both sides of 24 chunks per event,
where its blocks become wide, and of the 1,024 chunks of a round of theirs, with
small and empty events beside.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)


@pytest.mark.parametrize("sizes", [(24 * 4096 - 4096,), (24 * 4096 - 4095,), (1024 * 4096,), (1024 * 4096 + 1,), (5, 0, 1100 * 4096, 4097),
                                   (300000, 0, 7, 500000)])
def test_seed_numbers(cuda_lib, sizes):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    rng = np.random.default_rng(n)
    x, y = (rng.uniform(-245, 245, n).astype(np.float32) for _ in range(2))
    layer = np.concatenate([np.sort(rng.integers(0, 100, s)) for s in sizes]).astype(np.int32)
    w = rng.exponential(1.0, n).astype(np.float32)
    algo = C.Clusterizer(*PRM)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    assert_bitexact(got, oracle.clue2d_batch(off, x, y, layer, w, *PRM, n_threads=4))
