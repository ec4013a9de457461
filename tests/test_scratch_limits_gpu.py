"""Runs at the limits of the scratch budget.  A run needs `_bytes_2d` (the seed
bits, 512 bytes per chunk, are used where there is room beyond that): a budget of
exactly so much takes it, through every form of the call, beside CLUE3D and the
bridge on the same handle, in the pipelined host path and in a server.  Results
are the oracle's, or those of a handle with room, bit for bit."""
import numpy as np
import pytest

import clue_gb300 as C
import oracle
from clue_gb300 import synthetic as S

from _util import assert_bitexact

pytestmark = pytest.mark.gpu

PRM = (1.3, 2.0, 2.0)
KEYS = ("rho", "delta", "nearestHigher", "isSeed", "clusterIndex")
FIELDS = ("x", "y", "layer", "weight")


def _parts_2d(sizes, host):
    """The buffers that a run of up to three events (a tile table per layer) needs."""
    E, N = len(sizes), int(sum(sizes))
    chunks = int(sum((n + 4095) // 4096 for n in sizes))
    return [8 * (E + 1), 4 * (E + 1), 400 * E, 400 * E, 400 * E, 4 * N, 4 * N, 4 * N, 4 * N, 16 * N, 4 * N, 4 * N,
            4 * 10004 * 100 * E, 4 * chunks, 4 * chunks, 4 * chunks, 32, 4 * (100 * E + 512)] + ([16 * N, 20 * N] if host else [])


def _bytes_2d(sizes, host, held=False):
    """Their sum for a first run; `held`: as the arena holds them (multiples of 256 bytes)."""
    return sum((p + 255) // 256 * 256 if held else p for p in _parts_2d(sizes, host))


def _batch(sizes, seed, shuffled):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    ev = dict(x=rng.normal(0, 60, n).astype(np.float32), y=rng.normal(0, 60, n).astype(np.float32),
              layer=rng.integers(0, 100, n).astype(np.int32), weight=rng.exponential(1.0, n).astype(np.float32))
    if not shuffled:
        for e in range(len(sizes)):
            ev["layer"][off[e]:off[e + 1]].sort()
    return off, ev


def _run(algo, off, ev, flags):
    import torch
    if not flags & C.DEVICE_MEMORY:
        return algo.run_batch(off, *[ev[k] for k in FIELDS], flags=flags)
    n = int(off[-1])
    dev = {k: torch.from_numpy(ev[k]).cuda() for k in FIELDS}
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    torch.cuda.synchronize()
    algo.run_batch(off, *[dev[k] for k in FIELDS], out=out, flags=flags)
    algo.synchronize()
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("sizes", [(1,), (4097,), (200001,), (70000, 4096, 31), (150000, 0, 9000)])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("flags", [C.HOST_MEMORY, C.DEVICE_MEMORY, C.DEVICE_MEMORY | C.NO_GRAPH])
def test_budget_of_what_a_run_needs(cuda_lib, sizes, shuffled, flags):
    off, ev = _batch(sizes, len(sizes) + sizes[0], shuffled)
    want = oracle.clue2d_batch(off, *[ev[k] for k in FIELDS], *PRM, n_threads=4)
    need = _bytes_2d(sizes, not flags & C.DEVICE_MEMORY)
    algo = C.Clusterizer(*PRM, budget_bytes=need)
    assert_bitexact(_run(algo, off, ev, flags), want)
    algo.close()
    algo = C.Clusterizer(*PRM, budget_bytes=_bytes_2d(sizes, not flags & C.DEVICE_MEMORY, held=True))
    for _ in range(3):  # direct, captured, replayed
        assert_bitexact(_run(algo, off, ev, flags), want)
    algo.close()
    refused = C.Clusterizer(*PRM, budget_bytes=need - 8 * sum((n + 4095) // 4096 for n in sizes) - 1)
    with pytest.raises(C.ClueError) as ei:
        _run(refused, off, ev, flags)
    assert ei.value.code == C.CLUE_ENOMEM
    refused.close()


@pytest.mark.parametrize("flags", [C.PLAIN, C.PLAIN | C.DEVICE_MEMORY])
def test_plain_runs(cuda_lib, flags):
    sizes = (70000, 4096, 31)
    off, ev = _batch(sizes, 3, False)
    algo = C.Clusterizer(*PRM, budget_bytes=_bytes_2d((70000,), not flags & C.DEVICE_MEMORY) + 24 * len(sizes))
    got = _run(algo, off, ev, flags)
    algo.close()
    assert_bitexact(got, oracle.clue2d_batch(off, *[ev[k] for k in FIELDS], *PRM, n_threads=4))


def test_with_and_without_the_bits_in_turn(cuda_lib):
    """A handle whose budget has room for a small run's bits but not a large one's."""
    off1, ev1 = _batch((3000000,), 1, True)
    off2, ev2 = _batch((50000, 60000), 2, False)
    want1 = oracle.clue2d_batch(off1, *[ev1[k] for k in FIELDS], *PRM, n_threads=4)
    want2 = oracle.clue2d_batch(off2, *[ev2[k] for k in FIELDS], *PRM, n_threads=4)
    # the second run's tile tables (two events) stay in the arena
    algo = C.Clusterizer(*PRM, budget_bytes=_bytes_2d((3000000,), True, held=True) + 4 * 10004 * 100 + 8192)
    for _ in range(2):
        assert_bitexact(algo.run_batch(off1, *[ev1[k] for k in FIELDS]), want1)
        assert_bitexact(algo.run_batch(off2, *[ev2[k] for k in FIELDS]), want2)
    algo.close()


def test_beside_clue3d_and_the_bridge(cuda_lib):
    """The bits of a 2D run give way to CLUE3D and the bridge on the same handle."""
    import torch
    sizes = (400000, 200000)
    off, ev = _batch(sizes, 5, False)
    dev = {k: torch.from_numpy(ev[k]).cuda() for k in FIELDS}
    n = int(off[-1])
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    torch.cuda.synchronize()
    held = _bytes_2d(sizes, False, held=True)
    ev3 = S.clue3d_event(3, n_clusters=1000, n_layers=94)
    rows = 94 * 34 + 2
    need3 = 40 * rows + 148 * 1000 + 34 * 256  # the buffers of one event, host arrays
    algo = C.Clusterizer(*PRM, budget_bytes=held + need3)
    for _ in range(2):
        algo.run_batch(off, *[dev[k] for k in FIELDS], out=out, flags=C.DEVICE_MEMORY)
        got3, nts = algo.run_clue3d(np.array([0, 1000], np.int64), ev3)
        want3, nt = oracle.clue3d(ev3)
        assert int(nts[0]) == nt and np.array_equal(got3["tracksterIndex"], want3["tracksterIndex"])
    algo.close()
    assert_bitexact({k: v.cpu().numpy() for k, v in out.items()},
                    oracle.clue2d_batch(off, *[ev[k] for k in FIELDS], *PRM, n_threads=4))
    free = C.Clusterizer(*PRM)
    coff, want = free.layer_clusters(off, *[dev[k] for k in FIELDS], out)
    free.close()
    clusters = int(coff[-1])
    need_b = 16 * 3 + 4 * 100 + 4 * ((n + 4095) // 4096) + 8 + 28 * clusters + 32 + 9 * 256
    algo = C.Clusterizer(*PRM, budget_bytes=held + need_b)
    algo.run_batch(off, *[dev[k] for k in FIELDS], out=out, flags=C.DEVICE_MEMORY)
    coff2, got = algo.layer_clusters(off, *[dev[k] for k in FIELDS], out)
    algo.close()
    assert np.array_equal(coff, coff2)
    for k in want:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("sizes,slot", [((9000000, 9000000), (9000000,)),
                                        ((4000000, 3450000, 1100000, 12000000), (4000000, 3450000, 4550000)),
                                        ((1000000,) * 24, (1000000,) * 4)])
def test_pipelined_host_batches(cuda_lib, sizes, slot):
    """Two slots of a sub-batch each; the second case ends on a larger sub-batch
    in thirds and sixths of the batch (1.1 + 12M points) than in pieces of 8M (12M),
    the third has room for sixths only."""
    off, ev = _batch(sizes, 7, False)
    free = C.Clusterizer(*PRM)
    want = free.run_batch(off, *[ev[k] for k in FIELDS])
    free.close()
    algo = C.Clusterizer(*PRM, budget_bytes=2 * _bytes_2d(slot, True, held=True))
    got = algo.run_batch(off, *[ev[k] for k in FIELDS])
    algo.close()
    assert_bitexact(got, want)


def test_server_takes_its_largest_event_beside_a_used_slot(cuda_lib):
    """The largest event that the start-up buffers leave room for goes while the
    other slot, which has served events, holds its bits."""
    srv = C.Server(*PRM, budget_bytes=96 << 20, max_inflight=2, max_batch_events=4)
    cap = int(srv.stats()["slot_capacity_points"])
    for seed in range(6):
        off, ev = _batch((20000,) * 3, seed, True)
        for rid, out in srv.submit_many(off, *[ev[k] for k in FIELDS]):
            assert srv.poll(rid, timeout_ms=60000)[0] == C.CLUE_OK
    off, ev = _batch((cap,), 9, True)
    want = oracle.clue2d_batch(off, *[ev[k] for k in FIELDS], *PRM, n_threads=4)
    for _ in range(2):
        rid, out = srv.submit(*[ev[k] for k in FIELDS])
        assert srv.poll(rid, timeout_ms=60000)[0] == C.CLUE_OK
        assert_bitexact(out, want)
        off2, ev2 = _batch((20000,) * 3, 11, True)
        want2 = oracle.clue2d_batch(off2, *[ev2[k] for k in FIELDS], *PRM, n_threads=4)
        for e, (rid, out) in enumerate(srv.submit_many(off2, *[ev2[k] for k in FIELDS])):
            assert srv.poll(rid, timeout_ms=60000)[0] == C.CLUE_OK
            assert_bitexact(out, {k: v[off2[e]:off2[e + 1]] for k, v in want2.items()})
    srv.close()
