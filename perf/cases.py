"""Workloads on which this framework's speed is measured.

Each case is one call pattern of the public Python front end (which is a thin
binding of the C ABI): the clusterizer producer on one event from host or
device memory, batches of events on the device and from pinned host memory,
a burst into the serving loop, CLUE3D on layer clusters, and the 2D -> 3D
bridge.  Event shapes are the repository's: the toy-detector event (100
layers x (20 blobs x 40 points + 200 noise points)), HGCAL occupancy (100
layers x (50 blobs of 30..80 points + 500 noise points)), batches of uneven
events with sizes log-uniform in [5k, 200k], and CLUE3D events of 2k..20k
layer clusters.  Inputs are drawn on the GPU from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "heterogeneous-clue_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

LAYERS = 100
SIZES = 7  # seed of the sizes of events and blobs
FLT_MAX = float(np.finfo(np.float32).max)
POINT_FIELDS = ("x", "y", "layer", "weight")
FIELDS_3D = ("z", "eta", "phi", "r_over_absz", "radius", "layer", "energy", "isSilicon")


# ----------------------------------------------------------------- the cases

def listed():
    return [
        # The producer on the smallest event of the workloads, host arrays in
        # and out: what a framework module does per event; latency and launches.
        dict(name="event_5k_host", kind="event", memory="host", shape="uneven", lo=5000, hi=5000, shuffle=False,
             dc=1.3, rhoc=2.0, odf=2.0),
        # The same producer with device-resident points (the CUDA producer's
        # shape) on the toy-detector event, 100,000 points.
        dict(name="event_toy_device", kind="event", memory="device", shape="toy", lo=0, hi=0, shuffle=False,
             dc=1.3, rhoc=2.0, odf=2.0),
        # The reference's own shipped configuration (dc 20 cm, rhoc 25): search
        # boxes of many tiles, hundreds of neighbours per point.
        dict(name="event_toy_wide_device", kind="event", memory="device", shape="toy", lo=0, hi=0, shuffle=False,
             dc=20.0, rhoc=25.0, odf=2.0),
        # One HGCAL-occupancy event (about 325k points) whose points are not
        # grouped by layer, host arrays in and out: the largest producer call.
        dict(name="event_hgcal_shuffled_host", kind="event", memory="host", shape="hgcal", lo=0, hi=0, shuffle=True,
             dc=1.3, rhoc=2.0, odf=2.0),
        # A batch as a program assembles it from what has arrived: 48 uneven
        # events (about 2.5M points) on the device.
        dict(name="batch_48_device", kind="batch", memory="device", shape="uneven", events=48, lo=5000, hi=200000,
             shuffle=False, dc=1.3, rhoc=2.0, odf=2.0),
        # The headline batch: 4096 uneven events, 216M points, on the device.
        dict(name="batch_4096_device", kind="batch", memory="device", shape="uneven", events=4096, lo=5000, hi=200000,
             shuffle=False, dc=1.3, rhoc=2.0, odf=2.0),
        # HGCAL occupancy in a batch (dense layers of about 3,250 points).
        dict(name="batch_hgcal_200_device", kind="batch", memory="device", shape="hgcal", events=200, lo=0, hi=0,
             shuffle=False, dc=1.3, rhoc=2.0, odf=2.0),
        # End to end from pinned host memory, overlapped copies (27M points).
        dict(name="batch_512_host", kind="batch", memory="host", shape="uneven", events=512, lo=5000, hi=200000,
             shuffle=False, dc=1.3, rhoc=2.0, odf=2.0),
        # A burst of 12 uneven events into the serving loop, until all are back.
        dict(name="serve_burst_12", kind="serve", memory="host", shape="uneven", events=12, lo=5000, hi=200000,
             shuffle=False, dc=1.3, rhoc=2.0, odf=2.0),
        # CLUE3D on one event of layer clusters with the reference's default
        # parameters (94 layers, 3 sibling layers), host arrays in and out.
        dict(name="clue3d_event_host", kind="clue3d", memory="host", events=1, lo=5000, hi=5000, n_layers=94,
             siblings=3, critical_density=0.6),
        # The CLUE3D batch: 1,000 events of 2k..20k layer clusters, 100 layers.
        dict(name="clue3d_1000_device", kind="clue3d", memory="device", events=1000, lo=2000, hi=20000, n_layers=100,
             siblings=2, critical_density=0.5),
        # The bridge on 200 clustered HGCAL-occupancy events (65M points).
        dict(name="bridge_200_device", kind="bridge", memory="device", shape="hgcal", events=200, lo=0, hi=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the same kinds, sizes log-uniform over the same ranges."""
    kind = rng.choice(["event", "event", "batch", "batch", "batch_host", "serve", "clue3d", "clue3d", "bridge"])
    std = dict(dc=1.3, rhoc=2.0, odf=2.0)
    if kind == "event":
        prm = dict(std)
        if rng.random() < 0.25:
            prm = dict(dc=round(rng.uniform(0.8, 6.0), 3), rhoc=round(rng.uniform(1.0, 10.0), 3),
                       odf=round(rng.uniform(1.0, 2.5), 3))
        n = _log_int(rng, 5000, 325000)
        return dict(kind="event", memory=rng.choice(["host", "device"]), shape="uneven", lo=n, hi=n,
                    shuffle=rng.random() < 0.4, **prm)
    if kind == "batch":
        lo = _log_int(rng, 5000, 60000)
        return dict(kind="batch", memory="device", shape="uneven", events=_log_int(rng, 2, 3000), lo=lo,
                    hi=_log_int(rng, lo, 200000), shuffle=rng.random() < 0.3, **std)
    if kind == "batch_host":
        return dict(kind="batch", memory="host", shape="uneven", events=_log_int(rng, 2, 512), lo=5000, hi=200000,
                    shuffle=False, **std)
    if kind == "serve":
        return dict(kind="serve", memory="host", shape="uneven", events=_log_int(rng, 1, 12), lo=5000, hi=200000,
                    shuffle=rng.random() < 0.3, **std)
    if kind == "clue3d":
        lo = _log_int(rng, 2000, 20000)
        memory = rng.choice(["host", "device"])
        wide = rng.random() < 0.5
        return dict(kind="clue3d", memory=memory, events=_log_int(rng, 1, 1000 if memory == "device" else 50), lo=lo,
                    hi=_log_int(rng, lo, 20000), n_layers=94 if wide else 100, siblings=3 if wide else 2,
                    critical_density=0.6 if wide else 0.5)
    return dict(kind="bridge", memory="device", shape="uneven", events=_log_int(rng, 1, 400), lo=5000, hi=200000)


# -------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _points(case, seed):
    """Events of the case on the GPU: Gaussian blobs of hits on a uniform noise
    floor, layer by layer (blob points, then noise) unless shuffled.  Also
    which blob each point belongs to and whether it is noise.  Event and blob
    sizes belong to the case, everything else comes from the seed."""
    g, g_sizes = _gen(seed), _gen(SIZES)
    dev = "cuda"
    E = int(case.get("events", 1))
    if case["shape"] == "toy":
        nb, nn = np.full(E, 20, np.int64), np.full(E, 200, np.int64)
    elif case["shape"] == "hgcal":
        nb, nn = np.full(E, 50, np.int64), np.full(E, 500, np.int64)
    else:
        u = np.random.default_rng(SIZES).uniform(math.log(case["lo"]), math.log(case["hi"]), E)
        per_layer = np.exp(u) / LAYERS
        nn = np.rint(0.15 * per_layer).astype(np.int64)
        nb = np.maximum(np.rint((per_layer - nn) / 55.0), 0).astype(np.int64)
    G = E * LAYERS
    # one entry per blob and a last one for the noise of each (event, layer)
    per_group = torch.from_numpy(np.repeat(nb + 1, LAYERS)).to(dev)
    last = torch.cumsum(per_group, 0) - 1
    M = int(per_group.sum())
    group = torch.repeat_interleave(torch.arange(G, device=dev), per_group)
    noise = torch.zeros(M, dtype=torch.bool, device=dev)
    noise[last] = True
    if case["shape"] == "toy":
        size = torch.full((M,), 40, dtype=torch.int64, device=dev)
        sigma = torch.ones(M, device=dev)
    else:
        size = torch.randint(30, 81, (M,), generator=g_sizes, device=dev)
        sigma = 0.7 + 0.8 * torch.rand(M, generator=g, device=dev)
    size[last] = torch.from_numpy(np.repeat(nn, LAYERS)).to(dev)
    cx = 400.0 * torch.rand(M, generator=g, device=dev) - 200.0
    cy = 400.0 * torch.rand(M, generator=g, device=dev) - 200.0
    entry = torch.repeat_interleave(torch.arange(M, device=dev), size)
    n = entry.numel()
    is_noise = noise[entry]

    def coord(c):
        v = torch.randn(n, generator=g, device=dev) * sigma[entry] + c[entry]
        return torch.where(is_noise, 500.0 * torch.rand(n, generator=g, device=dev) - 250.0, v)

    x, y = coord(cx), coord(cy)
    w = torch.exp(0.5 * torch.randn(n, generator=g, device=dev))
    w = torch.where(is_noise, -0.1 * torch.log1p(-torch.rand(n, generator=g, device=dev)), w)
    gp = group[entry]
    layer = (gp % LAYERS).to(torch.int32)
    event = gp // LAYERS
    off = np.zeros(E + 1, np.int64)
    np.cumsum(torch.bincount(event, minlength=E).cpu().numpy(), out=off[1:])
    pts = dict(x=x, y=y, layer=layer, weight=w)
    if case.get("shuffle"):
        perm = torch.argsort(torch.rand(n, generator=g, device=dev), stable=True)
        perm = perm[torch.argsort(event[perm], stable=True)]
        pts = {k: v[perm].contiguous() for k, v in pts.items()}
    return off, pts, dict(entry=entry, is_noise=is_noise, event=event, g=g)


def _clusters3d(case, seed):
    """Layer clusters: eta U[1.5, 3.0], phi U[-pi, pi], energy LogNormal(0,
    0.7), a uniform layer; z from a 320..520 cm layer table, r/|z| = 1/sinh(eta)."""
    g = _gen(seed)
    E = int(case["events"])
    sizes = np.random.default_rng(SIZES).integers(case["lo"], case["hi"] + 1, E).astype(np.int64)
    off = np.zeros(E + 1, np.int64)
    np.cumsum(sizes, out=off[1:])
    n = int(off[-1])
    L = int(case["n_layers"])
    r = lambda: torch.rand(n, generator=g, device="cuda")  # noqa: E731
    eta = 1.5 + 1.5 * r()
    layer = torch.randint(0, L, (n,), generator=g, device="cuda").to(torch.int32)
    table = (320.0 + 200.0 * torch.arange(L, device="cuda", dtype=torch.float64) / (L - 1)).float()
    return off, dict(z=table[layer.long()], eta=eta, phi=math.pi * (2.0 * r() - 1.0),
                     r_over_absz=(1.0 / torch.sinh(eta.double())).float(),
                     radius=torch.full((n,), 2.0, device="cuda"), layer=layer,
                     energy=torch.exp(0.7 * torch.randn(n, generator=g, device="cuda")),
                     isSilicon=torch.ones(n, dtype=torch.int32, device="cuda"))


def _clustered(case, seed):
    """Points with a clustering as the 2D stage leaves it: a cluster per blob
    (ids in index order, its seed the blob's first point), one noise point in
    ten attached to a blob of its event, the others without a cluster."""
    off, pts, info = _points(case, seed)
    entry, noise, event = info["entry"], info["is_noise"], info["event"]
    blob_first = torch.ones_like(noise)
    blob_first[1:] = entry[1:] != entry[:-1]
    seed_pt = blob_first & ~noise
    rank = torch.cumsum(seed_pt.long(), 0) - 1
    per_event = torch.bincount(event[seed_pt], minlength=off.size - 1)
    base = torch.cumsum(per_event, 0) - per_event
    ci = rank - base[event]
    attach = torch.rand(entry.numel(), generator=info["g"], device="cuda") < 0.1
    ci = torch.where(noise & ~attach, -1, ci).clamp_(min=-1)
    out2d = dict(isSeed=seed_pt.to(torch.int32), clusterIndex=ci.to(torch.int32))
    return off, pts, out2d


_STREAM = []


def _stream():
    """The program's stream: every device-memory call is queued on it."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


def _outputs(n, spec, pinned=False):
    return {k: torch.empty(n, dtype=t, pin_memory=True) if pinned else torch.empty(n, dtype=t, device="cuda")
            for k, t in spec.items()}


SPEC_2D = dict(rho=torch.float32, delta=torch.float32, nearestHigher=torch.int32, isSeed=torch.int32,
               clusterIndex=torch.int32)
SPEC_3D = dict(rho=torch.float32, delta_transverse=torch.float32, delta_layers=torch.int32, nh_layer=torch.int32,
               nh_index=torch.int32, isSeed=torch.int32, tracksterIndex=torch.int32)


def prepare(case, seed):
    import clue_gb300 as C
    kind = case["kind"]
    st = dict(case=case, C=C)
    if kind == "clue3d":
        st["off"], pts = _clusters3d(case, seed)
        st["params"] = dict(n_layers=case["n_layers"], density_sibling_layers=case["siblings"],
                            nh_sibling_layers=case["siblings"], critical_density=case["critical_density"])
        st["algo"] = C.Clusterizer(1.3, 2.0, 2.0, stream=_stream() if case["memory"] == "device" else None)
        if case["memory"] == "host":
            st["pts"] = {k: v.cpu().numpy() for k, v in pts.items()}
        else:
            st["pts"] = pts
            st["out"] = _outputs(int(st["off"][-1]), SPEC_3D)
        return st
    if kind == "bridge":
        st["off"], st["pts"], st["out2d"] = _clustered(case, seed)
        st["algo"] = C.Clusterizer(1.3, 2.0, 2.0, stream=_stream())
        return st
    st["off"], pts, _ = _points(case, seed)
    if kind == "serve":
        st["srv"] = C.Server(case["dc"], case["rhoc"], case["odf"], budget_bytes=4 << 30)
        st["pts"] = {k: v.cpu().numpy() for k, v in pts.items()}
        return st
    st["algo"] = C.Clusterizer(case["dc"], case["rhoc"], case["odf"],
                               stream=_stream() if case["memory"] == "device" else None)
    if case["memory"] == "device":
        st["pts"], st["out"] = pts, _outputs(int(st["off"][-1]), SPEC_2D)
    elif kind == "event":
        st["pts"] = {k: v.cpu().numpy() for k, v in pts.items()}
    else:
        pinned = {k: torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v) for k, v in pts.items()}
        out = _outputs(int(st["off"][-1]), SPEC_2D, pinned=True)
        st["keep"] = (pinned, out)
        st["pts"] = {k: v.numpy() for k, v in pinned.items()}
        st["out"] = {k: v.numpy() for k, v in out.items()}
    return st


# ------------------------------------------------------------------- the run

def run(st):
    C, case, p = st["C"], st["case"], st["pts"]
    kind = case["kind"]
    flags = C.DEVICE_MEMORY if case["memory"] == "device" else C.HOST_MEMORY
    if kind == "clue3d":
        out, counts = st["algo"].run_clue3d(st["off"], p, params=st["params"], flags=flags, out=st.get("out"))
        return out if flags == C.DEVICE_MEMORY else dict(out, n_tracksters=counts)
    if kind == "bridge":
        coff, clusters = st["algo"].layer_clusters(st["off"], p["x"], p["y"], p["layer"], p["weight"], st["out2d"])
        return dict(clusters, cluster_offsets=coff)
    if kind == "serve":
        srv = st["srv"]
        reqs = srv.submit_many(st["off"], *[p[k] for k in POINT_FIELDS])
        srv.drain()
        for rid, _ in reqs:
            srv.poll(rid)
        return [o for _, o in reqs]
    if kind == "event" and case["memory"] == "host":
        return st["algo"].make_clusters(*[p[k] for k in POINT_FIELDS])
    return st["algo"].run_batch(st["off"], *[p[k] for k in POINT_FIELDS], out=st["out"], flags=flags)


# ------------------------------------------------------------ work, in bytes

def _n_points(case):
    """Expected points of a case."""
    E = case.get("events", 1)
    if case["shape"] == "toy":
        return 100000 * E
    if case["shape"] == "hgcal":
        return 325000 * E
    lo, hi = case["lo"], case["hi"]
    return E * (lo if lo == hi else (hi - lo) / math.log(hi / lo))


def work(case):
    """Each input read once, each output written once; the arithmetic of the
    pairs that lie inside the search radii (about 4 operations a pair)."""
    if case["kind"] == "clue3d":
        n = case["events"] * 0.5 * (case["lo"] + case["hi"])
        return dict(bytes=60.0 * n, flops=100.0 * n)
    n = _n_points(case)
    if case["kind"] == "bridge":
        clusters = 0.85 / 55 * n
        return dict(bytes=20.0 * n + 44.0 * clusters, flops=6.0 * n + 60.0 * clusters)
    # the toy event at dc 20 has about 16 + 64 noise points and a few blobs in the discs
    near = 55.0 if case["dc"] < 5 else 250.0
    return dict(bytes=36.0 * n, flops=4.0 * near * n)


# ------------------------------------------------- the same, in 64-bit floats

MOST_PAIRS = 4e10


def _layer_groups(off, layer):
    """Positions of each non-empty (event, layer), in index order, by size."""
    off_t = torch.from_numpy(off).cuda()
    n = layer.numel()
    ev = torch.searchsorted(off_t, torch.arange(n, device="cuda"), right=True) - 1
    key = ev * LAYERS + layer.long()
    order = torch.argsort(key, stable=True)
    cnt = torch.bincount(key, minlength=(off.size - 1) * LAYERS)
    start = torch.cumsum(cnt, 0) - cnt
    return order, start, cnt


def _exact_2d(case, seed):
    """rho and delta of every point, by comparing all points of a layer."""
    off, pts, _ = _points(case, seed)
    order, start, cnt = _layer_groups(off, pts["layer"])
    if float((cnt.double() ** 2).sum()) > MOST_PAIRS:
        return None
    f32 = np.float32
    dc = float(f32(case["dc"]))
    dm = float(f32(f32(case["odf"]) * f32(case["dc"])))
    x, y, w = (pts[k].double() for k in ("x", "y", "weight"))
    rho, delta = torch.zeros_like(x), torch.full_like(x, FLT_MAX)
    by_size = torch.argsort(cnt, descending=True)
    cs = cnt[by_size].cpu().numpy()
    i = 0
    while i < cs.size and cs[i] > 0:
        m = int(cs[i])
        b = max(1, min(4096, int(1e8 // (m * m))))
        j = min(cs.size, i + b)
        while j > i + 1 and cs[j - 1] == 0:
            j -= 1
        grp = by_size[i:j]
        col = torch.arange(m, device="cuda")
        ok = col[None, :] < cnt[grp][:, None]
        idx = order[(start[grp][:, None] + col[None, :]).clamp_(max=order.numel() - 1)]
        gx, gy, gw = x[idx], y[idx], torch.where(ok, w[idx], 0.0)
        d = torch.sqrt((gx[:, :, None] - gx[:, None, :]) ** 2 + (gy[:, :, None] - gy[:, None, :]) ** 2)
        d = d.masked_fill_(~(ok[:, None, :] & ok[:, :, None]), math.inf)
        r = 0.5 * torch.where(d <= dc, gw[:, None, :], 0.0).sum(2) + 0.5 * gw
        higher = (r[:, None, :] > r[:, :, None]) | ((r[:, None, :] == r[:, :, None]) & (col[None, None, :] > col[None, :, None]))
        best = d.masked_fill_(~higher | (d > dm), math.inf).min(2).values
        rho[idx[ok]] = r[ok]
        delta[idx[ok]] = torch.where(torch.isinf(best), FLT_MAX, best)[ok]
        i = j
    out = dict(rho=rho, delta=delta, nearestHigher=None, isSeed=None, clusterIndex=None)
    if case["kind"] != "serve":
        return out
    return [{k: None if v is None else v[off[e]:off[e + 1]] for k, v in out.items()} for e in range(off.size - 1)]


def _exact_3d(case, seed):
    off, p = _clusters3d(case, seed)
    if float((np.diff(off).astype(np.float64) ** 2).sum()) > MOST_PAIRS / 10:
        return None
    L, sib = case["n_layers"], case["siblings"]
    half = L // 2
    n = int(off[-1])
    rho = torch.zeros(n, dtype=torch.float64, device="cuda")
    delta = torch.full_like(rho, FLT_MAX)
    pi32 = float(np.float32(math.pi))
    two_pi32 = float(np.float32(2 * math.pi))
    for e in range(off.size - 1):
        s = slice(int(off[e]), int(off[e + 1]))
        z, eta, phi, roa, en = (p[k][s].double() for k in ("z", "eta", "phi", "r_over_absz", "energy"))
        lay = p["layer"][s].long()
        # bins as the tiles define them (integers, from 32-bit products)
        eb = ((p["eta"][s].abs() - 1.5) * (34.0 / float(np.float32(3.2) - np.float32(1.5)))).long().clamp_(0, 33)
        pb = ((phi + math.pi) * float(np.float32(126 / math.pi * 0.5))).long()
        lo = torch.where(lay < half, (lay - sib).clamp(min=0), (lay - sib).clamp(min=half))
        lo_nh = torch.where(lay < half, (lay - sib).clamp(min=0), (lay - sib).clamp(min=half + 1))
        hi = torch.where(lay < half, (lay + sib).clamp(max=half - 1), (lay + sib).clamp(max=2 * half - 1))
        k = lay.numel()
        r_all = torch.empty(k, dtype=torch.float64, device="cuda")
        step = max(1, int(2e7 // k))
        for phase in (0, 1):
            for a in range(0, k, step):
                i = slice(a, min(a + step, k))
                dphi = phi[i, None] - phi[None, :]
                dphi = torch.where(dphi.abs() > pi32, dphi - torch.round(dphi / (2 * math.pi)) * two_pi32, dphi)
                r1 = roa[None, :] * z[i, None]
                d2 = ((roa * z)[i, None] - r1) ** 2 + (r1 * dphi) ** 2
                same = lay[None, :] == lay[i, None]
                dpb = (pb[None, :] - pb[i, None]).abs()
                reach = 2 - phase
                near = ((eb[None, :] - eb[i, None]).abs() <= reach) & ((dpb <= reach) | (dpb >= 126 - reach))
                near &= lay[None, :] <= hi[i, None]
                if phase == 0:
                    near &= lay[None, :] >= lo[i, None]
                    coef = torch.where(same, 0.0, float(np.float32(0.2)))
                    me = torch.arange(k, device="cuda")[None, :] == torch.arange(k, device="cuda")[i, None]
                    coef = torch.where(me, 1.0, coef)
                    r_all[i] = torch.where(near & (d2 < float(np.float32(3.24))), coef * en[None, :], 0.0).sum(1)
                else:
                    near &= (lay[None, :] >= lo_nh[i, None]) & ~same & (r_all[None, :] > r_all[i, None])
                    best = d2.masked_fill(~near, math.inf).min(1).values
                    delta[s][i] = torch.where(torch.isinf(best), FLT_MAX, torch.sqrt(best))
        rho[s] = r_all
    out = dict(rho=rho, delta_transverse=delta, delta_layers=None, nh_layer=None, nh_index=None, isSeed=None,
               tracksterIndex=None)
    return out if case["memory"] == "device" else dict(out, n_tracksters=None)


def _exact_bridge(case, seed):
    off, pts, out2d = _clustered(case, seed)
    n = int(off[-1])
    ev = torch.repeat_interleave(torch.arange(off.size - 1, device="cuda"), torch.from_numpy(np.diff(off)).cuda())
    is_seed = out2d["isSeed"].bool()
    per_event = torch.bincount(ev[is_seed], minlength=off.size - 1)
    base = torch.cumsum(per_event, 0) - per_event
    ci = out2d["clusterIndex"].long()
    has = ci >= 0
    gid = (base[ev] + ci)[has]
    K = int(per_event.sum())
    w = pts["weight"].double()[has]

    def total(v):
        return torch.zeros(K, dtype=torch.float64, device="cuda").index_add_(0, gid, v)

    energy = total(w)
    x = total(w * pts["x"].double()[has]) / energy
    y = total(w * pts["y"].double()[has]) / energy
    layer = torch.zeros(K, dtype=torch.int64, device="cuda")
    seeds = torch.arange(n, device="cuda")[is_seed]
    layer[(base[ev] + ci)[is_seed]] = pts["layer"].long()[seeds]
    z = (320.0 + 200.0 * torch.arange(LAYERS, device="cuda", dtype=torch.float64) / (LAYERS - 1)).float().double()[layer]
    r = torch.sqrt(x * x + y * y)
    return dict(x=x, y=y, z=z, eta=torch.asinh(z / r), phi=torch.atan2(y, x), r_over_absz=r / z.abs(),
                radius=torch.full_like(x, 2.0), layer=None, energy=energy, isSilicon=None, cluster_offsets=None)


def exact(case, seed):
    if case["kind"] == "clue3d":
        return _exact_3d(case, seed)
    if case["kind"] == "bridge":
        return _exact_bridge(case, seed)
    return _exact_2d(case, seed)
