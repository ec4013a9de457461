"""Host-memory runs from page-locked arrays that lie back to back, each in a block
of its own or all in one, and from back-to-back pageable arrays: above and below
the staging limit.  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)
OUT = (("rho", np.float32), ("delta", np.float32), ("nearestHigher", np.int32), ("isSeed", np.int32),
       ("clusterIndex", np.int32))
IN = (("x", np.float32), ("y", np.float32), ("layer", np.int32), ("weight", np.float32))


def _blocks(n, kind):
    """Byte arrays of 4 n bytes, back to back: nine in one block, or separate
    page-locked blocks of which as many as possible lie back to back."""
    import torch
    if kind == "pageable":
        whole = np.zeros(36 * n, np.uint8)
    elif kind == "one block":
        whole = torch.zeros(36 * n, dtype=torch.uint8, pin_memory=True).numpy()
    else:
        blocks = [torch.zeros(4 * n, dtype=torch.uint8, pin_memory=True).numpy() for _ in range(64)]
        blocks.sort(key=lambda b: b.ctypes.data)
        runs = [[blocks[0]]]
        for b in blocks[1:]:
            if b.ctypes.data == runs[-1][-1].ctypes.data + 4 * n:
                runs[-1].append(b)
            else:
                runs.append([b])
        runs.sort(key=len)
        return (runs[-1] + [b for r in runs[:-1] for b in r])[:9]
    return [whole[4 * n * k:4 * n * (k + 1)] for k in range(9)]


@pytest.mark.parametrize("kind", ["separate blocks", "one block", "pageable"])
@pytest.mark.parametrize("n", [4096, 16384, 32768, 65536, 262144, 1 << 20])
def test_back_to_back_arrays(cuda_lib, kind, n):
    rng = np.random.default_rng(n)
    side = max(20.0, n ** 0.5 / 5)
    ev = dict(x=rng.uniform(-side, side, n).astype(np.float32), y=rng.uniform(-side, side, n).astype(np.float32),
              layer=np.sort(rng.integers(0, 100, n)).astype(np.int32), weight=rng.exponential(1.0, n).astype(np.float32))
    blocks = _blocks(n, kind)
    host = {}
    for (k, t), b in zip(IN, blocks):
        host[k] = b.view(t)
        host[k][:] = ev[k]
    out = {k: b.view(t) for (k, t), b in zip(OUT, blocks[4:])}
    want = oracle.clue2d(*[ev[k] for k, _ in IN], *PRM)
    for flags in (C.HOST_MEMORY, C.NO_GRAPH):
        algo = C.Clusterizer(*PRM)
        for _ in range(3):
            for v in out.values():
                v[:] = 77
            algo.run_batch(np.array([0, n], np.int64), *[host[k] for k, _ in IN], out=out, flags=flags)
            assert_bitexact(out, want)
        algo.close()
