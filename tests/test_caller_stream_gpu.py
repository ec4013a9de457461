"""Ordered batches (layers of both size classes, whose two passes run side by
side) on a caller's stream: they follow the work queued there before and
precede the work queued after, and every kernel has that stream's priority, also
after the handle has moved to another stream.  The priorities are read from the
kernel nodes of a captured run; nothing of it is launched."""
import ctypes

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


def _device(b):
    import torch
    n = int(b["offsets"][-1])
    dev = {k: torch.from_numpy(np.ascontiguousarray(b[k])).cuda() for k in FIELDS}
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    torch.cuda.synchronize()
    return dev, out


def _run(algo, b, dev, out, flags=0):
    algo.run_batch(b["offsets"], *[dev[k] for k in FIELDS], out=out, flags=C.DEVICE_MEMORY | flags)


def _captured_priorities(algo, stream, b, dev, out):
    """Priorities of the kernels of one run on `stream` (driver API)."""
    cu = ctypes.CDLL("libcuda.so.1")
    s, graph, n = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert cu.cuStreamBeginCapture_v2(s, 2) == 0  # CU_STREAM_CAPTURE_MODE_RELAXED
    try:
        _run(algo, b, dev, out, C.NO_GRAPH)
    finally:
        assert cu.cuStreamEndCapture(s, ctypes.byref(graph)) == 0
    with pytest.raises(C.ClueError):  # the run was captured: there is nothing to wait for
        algo.synchronize()
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    got = []
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:  # a kernel
            value = (ctypes.c_int * 16)()
            assert cu.cuGraphKernelNodeGetAttribute(ctypes.c_void_p(node), 8, value) == 0  # CU_LAUNCH_ATTRIBUTE_PRIORITY
            got.append(value[0])
    assert cu.cuGraphDestroy(graph) == 0
    return got


def test_kernels_have_the_callers_priority(cuda_lib):
    import torch
    b = S.uneven_batch(40, seed=3, lo=5000, hi=120000)
    dev, out = _device(b)
    high, low = torch.cuda.Stream(priority=-1), torch.cuda.Stream(priority=0)
    algo = C.Clusterizer(*PRM, stream=high.cuda_stream)
    for stream, priority in ((high, -1), (low, 0), (high, -1)):
        algo.set_stream(stream.cuda_stream)
        _run(algo, b, dev, out, C.NO_GRAPH)
        algo.synchronize()
        got = _captured_priorities(algo, stream, b, dev, out)
        assert len(got) == 10 and set(got) == {priority}, got
    algo.close()


@pytest.mark.parametrize("events", [30, 100])
def test_work_before_and_after(cuda_lib, events):
    """Inputs filled, and outputs read, by copies queued on the run's stream."""
    import torch
    batches = [S.uneven_batch(events, seed=s, lo=5000, hi=60000) for s in (5, 6)]
    want = [oracle.clue2d_batch(b["offsets"], *[b[k] for k in FIELDS], *PRM, n_threads=8) for b in batches]
    n = max(int(b["offsets"][-1]) for b in batches)
    fills = [_device(b)[0] for b in batches]
    dev = {k: torch.zeros(n, dtype=v.dtype, device="cuda") for k, v in fills[0].items()}
    out = {k: torch.empty(n, dtype=torch.float32 if k in ("rho", "delta") else torch.int32, device="cuda") for k in KEYS}
    a, c = (torch.zeros(1 << 28, dtype=torch.float32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    algo = C.Clusterizer(*PRM, stream=stream.cuda_stream)
    got = []
    for _ in range(3):
        for b, fill in zip(batches, fills):
            m = int(b["offsets"][-1])
            with torch.cuda.stream(stream):
                c.copy_(a)
                for k in FIELDS:
                    dev[k][:m].copy_(fill[k])
            _run(algo, b, dev, out)
            with torch.cuda.stream(stream):
                got.append({k: v[:m].clone() for k, v in out.items()})
    algo.synchronize()
    torch.cuda.synchronize()
    algo.close()
    for i, g in enumerate(got):
        assert_bitexact({k: v.cpu().numpy() for k, v in g.items()}, want[i % 2], label=f"run {i}")
