"""The bridge's fixed-point sums at the values where its conversions change
form: ties, products around 2^23 / 2^24 / 2^30 units (where the float product
loses its fraction, gains an even unit, and leaves the 32-bit conversion) and
denormals; runs that start, end and straddle event boundaries.  Bit-exact
against oracle/bridge.py (the sums are integers, so the tolerance is zero;
eta and phi as in the bridge's definition: 1 float ulp)."""
import numpy as np
import pytest

import clue_gb300 as C
from clue_gb300 import synthetic as S
from oracle import bridge as OB

from _util import max_ulp

pytestmark = pytest.mark.gpu


def _values(kind, rng, n):
    if kind == "ties":  # products that are odd multiples of half a unit of 2^-16, and neighbours
        w = np.ldexp(rng.integers(1, 2048, n).astype(np.float32), -rng.integers(0, 16, n))
        x = np.ldexp((2 * rng.integers(-2000, 2000, n) + 1).astype(np.float32), -rng.integers(0, 18, n))
    elif kind == "edges":  # |w * x| * 2^16 within a few ulps of powers of two from 2^20 to 2^33
        w = (1 + rng.integers(0, 1 << 23, n) * 2.0 ** -23).astype(np.float32)
        target = np.ldexp(1.0, rng.integers(4, 18, n)) * (1 + rng.integers(-4, 5, n) * 2.0 ** -24)
        x = (np.where(rng.random(n) < 0.5, -1, 1) * target / w).astype(np.float32)
    elif kind == "heavy":  # weights of 64 units of energy and more
        w = (64 * (1 + 4 * rng.random(n))).astype(np.float32)
        x = rng.uniform(-250, 250, n).astype(np.float32)
    else:  # tiny and denormal weights beside ordinary ones
        w = np.where(rng.random(n) < 0.5, np.ldexp(rng.random(n), -rng.integers(20, 149, n)), rng.random(n)).astype(np.float32)
        x = rng.uniform(-250, 250, n).astype(np.float32)
    return w, x


@pytest.mark.parametrize("per_cluster", [1, 3, 40])
@pytest.mark.parametrize("kind", ["ties", "edges", "heavy", "tiny"])
def test_fixed_point_forms(cuda_lib, kind, per_cluster):
    import torch
    rng = np.random.default_rng(len(kind) + per_cluster)
    sizes = np.array([1, 4095, 0, 17, 4097, 16, 6003], np.int64)  # boundaries inside and between runs of 16
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    w, x = _values(kind, rng, n)
    _, y = _values(kind, rng, n)
    local = np.concatenate([np.arange(s) for s in sizes])
    ci = (local // per_cluster).astype(np.int32)
    seed = (local % per_cluster == 0).astype(np.int32)
    ci[(local % per_cluster != 0) & (rng.random(n) < 0.2)] = -1
    layer = (local % 100).astype(np.int32)
    want_off, want = OB.layer_clusters(off, x, y, layer, w, seed, ci, S.layer_z())
    d = {k: torch.from_numpy(v).cuda() for k, v in dict(x=x, y=y, layer=layer, weight=w).items()}
    o2 = dict(isSeed=torch.from_numpy(seed).cuda(), clusterIndex=torch.from_numpy(ci).cuda())
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    got_off, got = algo.layer_clusters(off, d["x"], d["y"], d["layer"], d["weight"], o2)
    got = {k: v.cpu().numpy() for k, v in got.items()}
    algo.close()
    assert np.array_equal(got_off, want_off)
    for k, v in want.items():
        if k in ("eta", "phi"):
            assert max_ulp(got[k], v) <= 1, k
        else:
            assert np.array_equal(got[k].view(np.int32), np.asarray(v).view(np.int32)), k


@pytest.mark.parametrize("place", ["ring", "axes", "diagonal", "centre", "far"])
def test_cluster_fields_over_their_ranges(cuda_lib, place):
    """Positions and layer depths on both sides of every limit between the
    two-float and the double forms: signs, the axes, equal coordinates, clusters
    near the beam and far out, z negative, small against r, tiny and huge, and
    clusters without weight."""
    import torch
    rng = np.random.default_rng(len(place))
    n = 6000
    phi = rng.uniform(-np.pi, np.pi, n)
    r = {"ring": rng.uniform(20, 250, n), "axes": rng.uniform(0, 250, n), "diagonal": rng.uniform(1, 250, n),
         "centre": 10.0 ** rng.uniform(-9, 0, n), "far": 10.0 ** rng.uniform(2, 4, n)}[place]
    if place == "axes":
        phi = np.round(phi / (np.pi / 2)) * (np.pi / 2)
    if place == "diagonal":
        phi = (np.round(phi / (np.pi / 2)) + 0.5) * (np.pi / 2)
    x, y = (r * np.cos(phi)).astype(np.float32), (r * np.sin(phi)).astype(np.float32)
    if place == "axes":
        x[np.abs(x) < 1e-3] = 0
        y[np.abs(y) < 1e-3] = 0
    if place == "diagonal":
        y = np.copysign(np.abs(x), y)
    w = rng.exponential(1.0, n).astype(np.float32)
    w[rng.random(n) < 0.02] = 0
    lz = np.concatenate([S.layer_z(), -S.layer_z(), np.array([1e-4, 0.01, 1, 20, 60, 250, 1e5, 1e7, -5], np.float32)])
    lz = lz.astype(np.float32)
    layer = rng.integers(0, lz.size, n).astype(np.int32)
    ci = (np.arange(n) // 3).astype(np.int32)
    seed = (np.arange(n) % 3 == 0).astype(np.int32)
    off = np.array([0, n], np.int64)
    _, want = OB.layer_clusters(off, x, y, layer, w, seed, ci, lz)
    d = {k: torch.from_numpy(v).cuda() for k, v in dict(x=x, y=y, layer=layer, weight=w).items()}
    o2 = dict(isSeed=torch.from_numpy(seed).cuda(), clusterIndex=torch.from_numpy(ci).cuda())
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    _, got = algo.layer_clusters(off, d["x"], d["y"], d["layer"], d["weight"], o2, layer_z=lz)
    got = {k: v.cpu().numpy() for k, v in got.items()}
    algo.close()
    for k, v in want.items():
        if k in ("eta", "phi"):
            assert max_ulp(got[k], v) <= 1, k
        else:
            assert np.array_equal(got[k].view(np.int32), np.asarray(v).view(np.int32)), k


@pytest.mark.parametrize("shift", [8, 4, 1], ids=["32-byte", "16-byte", "4-byte"])
def test_alignments_of_the_inputs(cuda_lib, shift):
    """Arrays that start on a 32-byte, a 16-byte and a 4-byte boundary: each has
    its own loads."""
    import torch
    rng = np.random.default_rng(shift)
    off = np.array([0, 33, 8200], np.int64)
    n = int(off[-1])
    w, x = _values("heavy", rng, n)
    _, y = _values("edges", rng, n)
    local = np.concatenate([np.arange(s) for s in np.diff(off)])
    ci = (local // 5).astype(np.int32)
    seed = (local % 5 == 0).astype(np.int32)
    layer = (local % 100).astype(np.int32)
    want_off, want = OB.layer_clusters(off, x, y, layer, w, seed, ci, S.layer_z())
    d = [torch.from_numpy(np.concatenate([np.zeros(shift, v.dtype), v])).cuda()[shift:]
         for v in (x, y, layer, w, seed, ci)]
    algo = C.Clusterizer(1.3, 2.0, 2.0)
    got_off, got = algo.layer_clusters(off, *d[:4], dict(isSeed=d[4], clusterIndex=d[5]))
    got = {k: v.cpu().numpy() for k, v in got.items()}
    algo.close()
    assert np.array_equal(got_off, want_off)
    for k, v in want.items():
        if k in ("eta", "phi"):
            assert max_ulp(got[k], v) <= 1, k
        else:
            assert np.array_equal(got[k].view(np.int32), np.asarray(v).view(np.int32)), k
