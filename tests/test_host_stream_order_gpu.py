"""Host-memory runs on a caller's stream read their inputs behind the work that
the caller queued there before the call, whatever their size: page-locked arrays
are filled by a copy that waits behind some milliseconds of other work.  2D and
CLUE3D, on both sides of the staging limit (32,768 points).  Bit-exact against
the oracle on the new contents."""
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


def _late_arrays(stream, old, new):
    """Page-locked arrays that hold `old` and are filled with `new` by copies
    queued on `stream` behind a few milliseconds of copies."""
    import torch
    host = {k: torch.from_numpy(np.ascontiguousarray(v)).pin_memory() for k, v in old.items()}
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in new.items()}
    a, b = (torch.zeros(1 << 28, dtype=torch.float32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(16):
            b.copy_(a, non_blocking=True)
        for k in host:
            host[k].copy_(dev[k], non_blocking=True)
    return host, (dev, a, b)


def _event(n, seed):
    rng = np.random.default_rng(seed)
    return dict(x=rng.normal(0, 20, n).astype(np.float32), y=rng.normal(0, 20, n).astype(np.float32),
                layer=np.sort(rng.integers(0, 100, n)).astype(np.int32),
                weight=rng.exponential(1.0, n).astype(np.float32))


@pytest.mark.parametrize("n", [5000, 32768, 32769])
def test_clue2d_reads_in_stream_order(cuda_lib, n):
    import torch
    new = _event(n, n)
    stream = torch.cuda.Stream()
    algo = C.Clusterizer(*PRM, stream=stream.cuda_stream)
    warm = _event(n, 1)
    algo.make_clusters(*[warm[k] for k in ("x", "y", "layer", "weight")])
    host, keep = _late_arrays(stream, _event(n, 2), new)
    got = algo.make_clusters(*[host[k].numpy() for k in ("x", "y", "layer", "weight")])
    algo.close()
    assert_bitexact(got, oracle.clue2d(new["x"], new["y"], new["layer"], new["weight"], *PRM))
    del keep


@pytest.mark.parametrize("n", [5000, 32768, 32769])
def test_clue3d_reads_in_stream_order(cuda_lib, n):
    import torch
    fields = ("z", "eta", "phi", "r_over_absz", "radius", "layer", "energy", "isSilicon")
    ev = lambda seed: {k: v for k, v in S.clue3d_event(seed, n_clusters=n, n_layers=94).items() if k in fields}  # noqa: E731
    new = ev(n)
    off = np.array([0, n], np.int64)
    stream = torch.cuda.Stream()
    algo = C.Clusterizer(*PRM)
    algo.set_stream(stream.cuda_stream)
    algo.run_clue3d(off, ev(1))
    host, keep = _late_arrays(stream, ev(2), new)
    out, nts = algo.run_clue3d(off, {k: v.numpy() for k, v in host.items()})
    algo.close()
    want, nt = oracle.clue3d(S.clue3d_event(n, n_clusters=n, n_layers=94))
    assert int(nts[0]) == nt
    assert_bitexact({NAMES[k]: v for k, v in out.items()}, want, keys=tuple(NAMES.values()))
    del keep
