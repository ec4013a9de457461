"""The streaming kernels of the 2D pipeline at the edges of their chunks and
16-byte loads: event sizes around 4,096 points, events starting at every
alignment, arrays that are not 16-byte aligned, and input whose only layer
decrease sits on a chunk's or a load's first point (missing it would treat the
event as grouped by layer).  Bit-exact against the oracle."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)
SIZES = (1, 3, 4095, 2, 4096, 0, 4097, 5, 8193, 12288, 7)
KEYS = ("rho", "delta", "nearestHigher", "isSeed", "clusterIndex")


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("decrease", [None, 1, 4, 4095, 4096, 4097, 8192, -1])
def test_chunk_and_load_edges(cuda_lib, shift, decrease):
    """decrease: the position, in every event that has it, of the one point
    whose layer is below its predecessor's; shift: the arrays' offset in words."""
    import torch
    rng = np.random.default_rng(3)
    off = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.int64)
    n = int(off[-1])
    x = rng.uniform(-30, 30, n).astype(np.float32)
    y = rng.uniform(-30, 30, n).astype(np.float32)
    w = rng.exponential(1.0, n).astype(np.float32)
    layer = np.empty(n, np.int32)
    for e, size in enumerate(SIZES):
        l = np.sort(rng.integers(1, 6, size)).astype(np.int32)
        at = size - 1 if decrease == -1 else decrease
        if at is not None and 0 < at < size:
            l[at] = 0
            l[at + 1:] = np.sort(l[at + 1:])
        layer[off[e]:off[e + 1]] = l
    dev = {}
    for k, v in dict(x=x, y=y, layer=layer, weight=w).items():
        t = torch.empty(n + shift, dtype=torch.from_numpy(v).dtype, device="cuda")
        t[shift:] = torch.from_numpy(v).cuda()
        dev[k] = t[shift:]
    out = {k: torch.empty(n + shift, dtype=torch.float32 if k in ("rho", "delta") else torch.int32,
                          device="cuda")[shift:] for k in KEYS}
    torch.cuda.synchronize()
    algo = C.Clusterizer(*PRM)
    algo.run_batch(off, dev["x"], dev["y"], dev["layer"], dev["weight"], out=out, flags=C.DEVICE_MEMORY)
    algo.synchronize()
    algo.close()
    want = oracle.clue2d_batch(off, x, y, layer, w, *PRM, n_threads=4)
    assert_bitexact({k: v.cpu().numpy() for k, v in out.items()}, want)


@pytest.mark.parametrize("n", [1023, 1025, 5121, 152 * 4096, 152 * 4096 + 1])
def test_shuffled_event_sizes(cuda_lib, n):
    """One event with its layers interleaved, around the slices of a chunk that
    a block of the grouping kernel takes, and on both sides of 152 chunks."""
    rng = np.random.default_rng(n)
    side = 30 + n ** 0.5 / 8
    x, y = (rng.uniform(-min(side, 200), min(side, 200), n).astype(np.float32) for _ in range(2))
    layer = rng.integers(0, 100, n).astype(np.int32)
    w = rng.exponential(1.0, n).astype(np.float32)
    algo = C.Clusterizer(*PRM)
    got = algo.make_clusters(x, y, layer, w)
    algo.close()
    assert_bitexact(got, oracle.clue2d(x, y, layer, w, *PRM))


@pytest.mark.parametrize("points", [12 << 20, (12 << 20) + 1])
def test_large_shuffled_batches(cuda_lib, points):
    """A shuffled batch on both sides of the size from which its layers are
    taken event by event, with layers of both size classes and an empty event."""
    rng = np.random.default_rng(points)
    sizes = rng.integers(20000, 260000, 90)
    sizes = np.concatenate([[0], (sizes * ((points - 300000) / sizes.sum())).astype(np.int64)])
    sizes = np.concatenate([sizes, [points - sizes.sum()]])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    x, y = (rng.uniform(-240, 240, points).astype(np.float32) for _ in range(2))
    layer = rng.integers(0, 100, points).astype(np.int32)
    w = rng.exponential(1.0, points).astype(np.float32)
    algo = C.Clusterizer(*PRM)
    got = algo.run_batch(off, x, y, layer, w)
    algo.close()
    assert_bitexact(got, oracle.clue2d_batch(off, x, y, layer, w, *PRM, n_threads=8))


@pytest.mark.parametrize("n", [1, 31, 4096, 32767, 32768, 32769])
def test_small_host_runs_and_the_rule(cuda_lib, n):
    """Host-memory runs on both sides of the staging limit (32,768 points),
    from read-only inputs, twice in a row (the second may replay a graph)."""
    rng = np.random.default_rng(n)
    ev = dict(x=rng.normal(0, 20, n).astype(np.float32), y=rng.normal(0, 20, n).astype(np.float32),
              layer=np.sort(rng.integers(0, 100, n)).astype(np.int32), weight=rng.exponential(1.0, n).astype(np.float32))
    for v in ev.values():
        v.flags.writeable = False
    want = oracle.clue2d(ev["x"], ev["y"], ev["layer"], ev["weight"], *PRM)
    algo = C.Clusterizer(*PRM)
    for _ in range(3):
        assert_bitexact(algo.make_clusters(ev["x"], ev["y"], ev["layer"], ev["weight"]), want)
    bad = np.array(ev["layer"])
    bad[-1] = 100
    with pytest.raises(C.ClueError, match="layer"):
        algo.make_clusters(ev["x"], ev["y"], bad, ev["weight"])
    assert_bitexact(algo.make_clusters(ev["x"], ev["y"], ev["layer"], ev["weight"]), want)
    algo.close()


@pytest.mark.parametrize("events", [8, 60])
@pytest.mark.parametrize("tuning", [(256, 1536, 512, 4096), (256, 500, 256, 900), (128, 64, 512, 128)])
def test_ordered_passes_side_by_side(cuda_lib, events, tuning):
    """Ordered batches whose layers fall into both classes, with a first capacity
    inside a size class and layers above both capacities (HBM scratch):
    repeated runs (direct, captured, replayed) give the oracle's bits."""
    import torch
    b = S.uneven_batch(events, seed=11, lo=5000, hi=180000)
    want = oracle.clue2d_batch(b["offsets"], b["x"], b["y"], b["layer"], b["weight"], *PRM, n_threads=8)
    n = int(b["offsets"][-1])
    dev = {k: torch.from_numpy(np.ascontiguousarray(b[k])).cuda() for k in ("x", "y", "layer", "weight")}
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    algo = C.Clusterizer(*PRM)
    algo.set_tuning(threads=tuning[0], layer_capacity=tuning[1], big_threads=tuning[2], big_capacity=tuning[3])
    for _ in range(3):
        for v in out.values():
            v.zero_()
        torch.cuda.synchronize()
        algo.run_batch(b["offsets"], dev["x"], dev["y"], dev["layer"], dev["weight"], out=out, flags=C.DEVICE_MEMORY)
        algo.synchronize()
        assert_bitexact({k: v.cpu().numpy() for k, v in out.items()}, want)
    algo.close()
