"""Shuffled batches around the numbers of chunks at which the grouping kernel's
grid changes (five chunks per SM) and its blocks begin to take chunks by ticket,
repeated.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)


@pytest.mark.parametrize("chunks_per_sm,extra", [(1, 1), (2, 1), (3, 0), (5, 0), (5, 1), (6, 1), (13, 0)])
def test_chunk_counts(cuda_lib, chunks_per_sm, extra):
    import torch
    chunks = chunks_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(chunks)
    # events of one to five chunks, most chunks not full
    per = []
    while sum(per) < chunks:
        per.append(min(int(rng.integers(1, 6)), chunks - sum(per)))
    sizes = [int(rng.integers((c - 1) * 4096 + 1, (c - 1) * 4096 + 1500)) for c in per]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    x, y = (rng.uniform(-200, 200, n).astype(np.float32) for _ in range(2))
    layer = rng.integers(0, 100, n).astype(np.int32)
    w = rng.exponential(1.0, n).astype(np.float32)
    want = oracle.clue2d_batch(off, x, y, layer, w, *PRM, n_threads=8)
    algo = C.Clusterizer(*PRM)
    for _ in range(3):
        assert_bitexact(algo.run_batch(off, x, y, layer, w), want)
    algo.close()
