"""The work a user has this engine do, as measurable cases.

Each case is one call sequence through the public entry points (the ctypes front end or the
C ABI behind it), over inputs with the distributions of the repository's own workloads
(gcmfgh.synth): star polygons in uniform or clustered layers, spiky single pairs, the
degeneracy-stressed batch, islands with holes, and serving bursts.

Results go into buffers of a fixed capacity that the program keeps, as one that calls the
C ABI has them.

Kinds:
  pair    two host rings clipped by one clip_pair call, results read to the host
  join    two device-resident layers: join, then clip of the join's clip set, results copied
          on the device
  mbr     two device-resident layers: the join alone, its per-candidate fields on the device
  host    two host layers (pinned): join + clip from host buffers, results back in host buffers
  batch   device-resident polygon pairs clipped by one clip_batch call (degenerate inputs)
  multi   host polygon pairs with several rings each (holes), one gh_clip_multi_batch call
  serve   a burst of query rings submitted to a running server, every result taken
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "gcmf-gh_b200"))
import gcmfgh  # noqa: E402
from gcmfgh import synth  # noqa: E402

_DEV = "cuda:0"
_JOIN_OUT = ("b", "o", "cmbr", "pip_flag", "seg_flag", "clip")


def listed():
    return [
        # one pair of hand-sized polygons, as the per-pair entry point is called in a loop:
        # launches and host round trips are all there is
        {"name": "pair_small", "kind": "pair", "np": 37, "nq": 24, "exact": False},
        # two very long rings crossing each other everywhere (a coastline against a detailed
        # mask); exact predicates, which such a pair needs
        {"name": "pair_large_exact", "kind": "pair", "np": 400_000, "nq": 200_000, "exact": True},
        # two small layers (2,000 x 2,000 stars of 8 to 64 vertices), an interactive overlay
        {"name": "join_small", "kind": "join", "shape": "uniform", "nb": 2000, "no": 2000, "exact": False, "union": False},
        # the batched overlay of two clustered layers with heavy-tailed vertex counts
        {"name": "join_batched", "kind": "join", "shape": "clustered", "nb": 200_000, "no": 200_000, "exact": False, "union": False},
        # a mid-sized ragged overlay, union of every joined pair
        {"name": "join_union", "kind": "join", "shape": "clustered", "nb": 61_003, "no": 23_501, "exact": False, "union": True},
        # a mid-sized overlay under exact predicates
        {"name": "join_exact", "kind": "join", "shape": "uniform", "nb": 30_011, "no": 40_009, "exact": True, "union": False},
        # the spatial join alone (candidates, containment and intersection flags)
        {"name": "join_only", "kind": "mbr", "shape": "clustered", "nb": 300_007, "no": 120_001},
        # the whole call from host layers to host results, as the reference's main() does it
        {"name": "host_to_host", "kind": "host", "shape": "clustered", "nb": 100_000, "no": 100_000},
        # degeneracy-stressed pairs, vertex counts to 10,000: shared vertices, collinear
        # overlaps, translations by 1e-12, in both precision modes
        {"name": "degenerate_exact", "kind": "batch", "n": 10_007, "vmax": 10_000, "exact": True},
        {"name": "degenerate_tolerance", "kind": "batch", "n": 6_001, "vmax": 10_000, "exact": False},
        # polygons of several islands with holes, a batch per call
        {"name": "multi_rings", "kind": "multi", "n": 3000, "vmin": 5, "vmax": 200},
        # a burst of queries against a resident layer
        {"name": "serve_burst", "kind": "serve", "resident": 200_000, "queries": 12, "qmax": 50_000},
    ]


def _mean_log(lo, hi):
    """The mean of a log-uniform size."""
    return (hi - lo) / math.log(hi / lo)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pair", "pair", "join", "join", "join", "mbr", "host", "batch", "batch", "multi", "serve"))
    if kind == "pair":
        np_ = _log_int(rng, 8, 400_000)
        nq = max(5, int(np_ * rng.uniform(0.1, 0.5)))
        # the tolerance is absolute, so long spiky rings are only meaningful exactly
        return {"kind": kind, "np": np_, "nq": nq, "exact": np_ > 2000 or rng.random() < 0.5}
    if kind in ("join", "mbr", "host"):
        top = {"join": 200_000, "mbr": 300_000, "host": 100_000}[kind]
        shape = rng.choice(("uniform", "clustered"))
        nb, no = (_log_int(rng, 500, top if shape == "clustered" else top // 4) for _ in range(2))
        c = {"kind": kind, "shape": shape, "nb": nb, "no": no}
        if kind == "join":
            c.update(exact=rng.random() < 0.3, union=rng.random() < 0.3)
        return c
    if kind == "batch":
        vmax = _log_int(rng, 200, 10_000)
        return {"kind": kind, "n": _log_int(rng, 60, 6_000), "vmax": vmax, "exact": rng.random() < 0.5}
    if kind == "multi":
        return {"kind": kind, "n": _log_int(rng, 10, 3000), "vmin": 5, "vmax": _log_int(rng, 20, 200)}
    return {"kind": kind, "resident": _log_int(rng, 10_000, 200_000), "queries": rng.randint(1, 12),
            "qmax": _log_int(rng, 1000, 50_000)}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(int(seed))
    return g


def _u(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, dtype=torch.float64, device=_DEV)


def _stars(g, counts, centres, base, rmin, rmax):
    """Star polygons as a layer (xy with closing vertices, vnum, vps), on the device:
    vertices at sorted uniform angles, radius base * U(rmin, rmax)."""
    n, total = counts.numel(), int(counts.sum())
    pid = torch.repeat_interleave(torch.arange(n, device=_DEV), counts)
    ang = _u(g, total, 0.0, 2.0 * math.pi)
    order = torch.argsort(ang)
    order = order[torch.argsort(pid[order], stable=True)]
    ang = ang[order]
    rad = base[pid] * _u(g, total, rmin, rmax)
    xy = torch.stack([centres[pid, 0] + rad * torch.cos(ang), centres[pid, 1] + rad * torch.sin(ang)], 1)
    vnum = counts + 1
    ends = torch.cumsum(vnum, 0)
    out = torch.empty(int(ends[-1]), 2, dtype=torch.float64, device=_DEV)
    out[torch.arange(total, device=_DEV) + pid] = xy
    out[ends - 1] = out[ends - vnum]
    return out.reshape(-1).contiguous(), vnum.to(torch.int32), ends


def _layer(g, shape, n, scale, means):
    """One layer of n stars.  uniform: 8 to 64 vertices, centres uniform; clustered:
    Pareto(1.5, 4) vertex counts capped at 100,000, centres from a Gaussian mixture.
    scale stretches the extent, so that the overlaps per polygon do not depend on the size."""
    z = torch.randn(n, 3, generator=g, dtype=torch.float64, device=_DEV)
    if shape == "uniform":
        counts = torch.randint(8, 65, (n,), generator=g, device=_DEV)
        centres = torch.stack([_u(g, n), _u(g, n)], 1) * (1000.0 * scale)
        return _stars(g, counts, centres, torch.exp(math.log(5.0) + 0.5 * z[:, 0]), 0.6, 1.0)
    counts = torch.clamp(torch.floor(4.0 * torch.pow(1.0 - _u(g, n), -1.0 / 1.5)), max=100_000).to(torch.int64)
    comp = torch.randint(0, means.shape[0], (n,), generator=g, device=_DEV)
    centres = means[comp] + 2000.0 * scale * z[:, 1:]
    return _stars(g, counts, centres, torch.exp(math.log(50.0) + 0.7 * z[:, 0]), 0.6, 1.0)


def _layers(case, seed):
    g = _generator(seed)
    full = 2000 if case["shape"] == "uniform" else 200_000
    scale = math.sqrt(max(case["nb"], case["no"]) / full)
    means = torch.stack([_u(g, 64), _u(g, 64)], 1) * (1e5 * scale)
    return _layer(g, case["shape"], case["nb"], scale, means), _layer(g, case["shape"], case["no"], scale, means)


def _pair_rings(case, seed):
    """Two concentric-ish spiky stars (open rings, host)."""
    g = _generator(seed)
    rings = []
    for n, c, lo, hi in ((case["np"], (0.0, 0.0), 0.8, 1.2), (case["nq"], (0.05, 0.03), 0.7, 1.3)):
        xy, _, _ = _stars(g, torch.tensor([n], device=_DEV), torch.tensor([c], dtype=torch.float64, device=_DEV),
                          torch.ones(1, dtype=torch.float64, device=_DEV), lo, hi)
        rings.append(xy[:-2].cpu().numpy())
    return rings


def _pinned_layer(t):
    """A host layer (synth.Layer over pinned memory) of device tensors."""
    xy, vnum, vps = (x.cpu().pin_memory() for x in t)
    host = synth.Layer(xy.numpy(), vnum.numpy())
    host.vps, host.keep = vps.numpy(), (xy, vnum, vps)
    return host


class _Server(gcmfgh.Server):
    """A server that is closed with the program's last reference to it."""

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


_TORCH = {np.int32: torch.int32, np.int64: torch.int64, np.float64: torch.float64, np.int8: torch.int8,
          np.uint8: torch.uint8}


def _capacity(case):
    """Elements of the result buffers a program sets aside for a case: several times what
    the workload gives, since the clustered layers' vertex counts are heavy-tailed."""
    kind = case["kind"]
    if kind == "pair":
        n = case["np"] + case["nq"]
        return {"status": 1, "ncomp": 1, "comp_size": 8 * n + 1024, "xy": 2 * (20 * n + 4096)}
    if kind in ("join", "mbr", "host"):
        m, uniform = min(case["nb"], case["no"]), case["shape"] == "uniform"
        if kind == "mbr":
            k = (4 if uniform else 16) * m + 65536
            return {name: 4 * k if name == "cmbr" else k for name in _JOIN_OUT}
        k = (2 if uniform else 8) * m + 4096
        v = (150 * m + 8_000_000) if case.get("union") else (50 * m + 4_000_000)
        c = {"status": k, "ncomp": k, "comp_size": 2 * k + 100_000, "xy": 2 * (v // 8 if uniform else v)}
        return {**c, "clip_b": k, "clip_o": k} if kind == "join" else c
    if kind == "batch":
        v = int(2 * _mean_log(4, case["vmax"]) * case["n"])
        return {"status": case["n"], "ncomp": case["n"], "comp_size": v + 50_000, "xy": 2 * (3 * v + 300_000)}
    if kind == "multi":
        n = case["n"]
        return {"status": n, "ncomp": n, "comp_size": 40 * n + 1000, "xy": 2 * (12 * case["vmax"] * n + 10_000)}
    return {"ids": 8192, "status": 8192, "ncomp": 8192, "comp_size": 65536, "xy": 2 * (20 * case["qmax"] + 200_000)}


def _fields(name):
    return gcmfgh.JOIN_FIELDS if name in gcmfgh.JOIN_FIELDS and name not in gcmfgh.CLIP_FIELDS else gcmfgh.CLIP_FIELDS


def _buffers(case, on_device):
    kw = {"device": _DEV} if on_device else {"pin_memory": True}
    return {name: torch.zeros(n, dtype=_TORCH[_fields(name)[name][1]], **kw) for name, n in _capacity(case).items()}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "serve":
        g = _generator(seed)
        scale = math.sqrt(case["resident"] / 200_000)
        means = torch.stack([_u(g, 64), _u(g, 64)], 1) * (1e5 * scale)
        xy, vnum, _ = _layer(g, "clustered", case["resident"], scale, means)
        s["server"] = _Server(synth.Layer(xy.cpu().numpy(), vnum.cpu().numpy()))
        n = case["queries"]
        counts = torch.exp(_u(g, n, math.log(16.0), math.log(case["qmax"] + 1.0))).to(torch.int64)
        z = torch.randn(n, 3, generator=g, dtype=torch.float64, device=_DEV)
        comp = torch.randint(0, 64, (n,), generator=g, device=_DEV)
        q = _stars(g, counts, means[comp] + 2000.0 * scale * z[:, 1:], torch.exp(math.log(50.0) + 0.7 * z[:, 0]), 0.6, 1.0)
        ql = synth.Layer(q[0].cpu().numpy(), q[1].cpu().numpy())
        s["rings"] = [np.ascontiguousarray(ql.ring(i)) for i in range(n)]
        s["out"] = [{name: np.zeros(c, np.float64 if name == "xy" else np.int32) for name, c in _capacity(case).items()}
                    for _ in range(n)]
        return s
    eng = s["engine"] = gcmfgh.Engine(0, union=case.get("union", False))
    eng.set_precision(case.get("exact", False))
    s["on_device"] = kind in ("join", "mbr", "batch")
    s["out"] = _buffers(case, s["on_device"])
    if kind == "pair":
        s["P"], s["Q"] = _pair_rings(case, seed)
    elif kind in ("join", "mbr"):
        s["base"], s["overlay"] = (gcmfgh.DeviceLayer.from_tensors(*t) for t in _layers(case, seed))
    elif kind == "host":
        s["base"], s["overlay"] = (_pinned_layer(t) for t in _layers(case, seed))
    elif kind == "batch":
        _, P, Q = synth.degeneracy_chunk_device(seed, 0, case["n"], _DEV, vmax=case["vmax"])
        s["base"], s["overlay"] = gcmfgh.DeviceLayer.from_tensors(*P), gcmfgh.DeviceLayer.from_tensors(*Q)
        s["ids"] = torch.arange(case["n"], dtype=torch.int32, device=_DEV)
    else:
        pairs = synth.holed_pairs(seed, case["n"], case["vmin"], case["vmax"])
        for side in (0, 1):
            rings = [r for pq in pairs for r in pq[side]]
            s["xy", side] = np.ascontiguousarray(np.concatenate([r.reshape(-1) for r in rings]))
            s["sizes", side] = np.array([len(r) for r in rings], np.int32)
            s["rings", side] = np.array([len(pq[side]) for pq in pairs], np.int32)
    return s


# ---------------------------------------------------------------- one pass
def _read(s):
    """The result fields, copied into the program's buffers."""
    lib, nb = gcmfgh.lib(), ctypes.c_int64()
    for name, t in s["out"].items():
        fields = _fields(name)
        getter = lib.gh_clip_get if fields is gcmfgh.CLIP_FIELDS else lib.gcmf_join_get
        gcmfgh._check(getter(s["engine"].h, fields[name][0], ctypes.c_void_p(t.data_ptr()), t.numel() * t.element_size(),
                             int(s["on_device"]), ctypes.byref(nb)))
    return s["out"]


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def run(s):
    kind = s["kind"]
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(r) for r in s["rings"]]
        for t, o in zip(tickets, s["out"]):
            info = srv.wait(t)
            if info["n_hits"] > len(o["ids"]) or info["n_components"] > len(o["comp_size"]) or 2 * info["n_vertices"] > len(o["xy"]):
                raise RuntimeError("result larger than its buffers")
            gcmfgh._check(gcmfgh.lib().gcmfgh_serve_take(srv.h, t, _ptr(o["ids"]), _ptr(o["status"]), _ptr(o["ncomp"]),
                                                         _ptr(o["comp_size"]), _ptr(o["xy"])))
        return s["out"]
    eng = s["engine"]
    if kind == "pair":
        eng.clip_pair(s["P"], s["Q"])
    elif kind in ("join", "mbr"):
        eng.join(s["base"], s["overlay"])
        if kind == "join":
            eng.clip_joined(s["base"], s["overlay"])
    elif kind == "host":
        eng.join_clip_host(s["base"], s["overlay"])
    elif kind == "batch":
        eng.clip_batch(s["base"], s["overlay"], s["ids"], s["ids"])
    else:
        info = gcmfgh.ClipInfo()
        gcmfgh._check(gcmfgh.lib().gh_clip_multi_batch(
            eng.h, len(s["rings", 0]), _ptr(s["xy", 0]), _ptr(s["sizes", 0]), _ptr(s["rings", 0]),
            _ptr(s["xy", 1]), _ptr(s["sizes", 1]), _ptr(s["rings", 1]), ctypes.byref(info)))
    return _read(s)


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Inputs read once, results written once; about 40 operations per intersection and 10
    per input vertex.  Counts are the distributions' means (the results per pair as the
    workloads give them)."""
    kind = case["kind"]
    if kind == "pair":
        vin, rec = case["np"] + case["nq"], 3.6e-4 * case["np"] * case["nq"]
        out, pairs = min(rec + 0.5 * vin, 9.0 * vin), 1      # slivers between long rings are tidied away
    elif kind in ("join", "mbr", "host"):
        uniform = case["shape"] == "uniform"
        vin = (37.0 if uniform else 11.5) * (case["nb"] + case["no"])
        pairs = (0.8 if uniform else 2.4) * min(case["nb"], case["no"])
        rec, out = (3.0 if uniform else 2.5) * pairs, (18.0 if uniform else 9.0) * pairs
        if kind == "mbr":
            rec, out, pairs = 0.0, 0.0, 3.6 * min(case["nb"], case["no"])
    elif kind == "batch":
        vin = 2 * _mean_log(4, case["vmax"]) * case["n"]
        rec, out, pairs = 0.9 * vin, 1.2 * vin, case["n"]
    elif kind == "multi":
        vin, pairs = 7.5 * 0.5 * (case["vmin"] + case["vmax"]) * 0.75 * case["n"], case["n"]
        rec, out = 0.1 * vin, 0.5 * vin
    else:
        vin = _mean_log(16, case["qmax"]) * case["queries"]
        rec, out, pairs = vin, 2.5 * vin, 17 * case["queries"]
    per_pair = 43 if kind == "mbr" else 16
    return {"bytes": 16.0 * vin + 16.0 * out + per_pair * pairs, "flops": 40.0 * rec + 10.0 * vin}


# ---------------------------------------------------------------- exact results, plain numpy
def _side(a, b, c):
    return (b[..., 0] - a[..., 0]) * (c[..., 1] - a[..., 1]) - (b[..., 1] - a[..., 1]) * (c[..., 0] - a[..., 0])


def _crossings(P, Q):
    """Properly crossing edge pairs of two rings: (P edge, Q edge, place on P, place on Q)."""
    P2, Q2 = np.roll(P, -1, 0), np.roll(Q, -1, 0)
    got, step = [], max(1, 2_000_000 // len(Q))
    for i in range(0, len(P), step):
        a, b = P[i:i + step, None], P2[i:i + step, None]
        s1, s2 = _side(Q[None], Q2[None], a), _side(Q[None], Q2[None], b)
        t1, t2 = _side(a, b, Q[None]), _side(a, b, Q2[None])
        p, q = np.nonzero((s1 * s2 < 0) & (t1 * t2 < 0))
        got.append((p + i, q, s1[p, q] / (s1[p, q] - s2[p, q]), t1[p, q] / (t1[p, q] - t2[p, q])))
    return tuple(np.concatenate(x) for x in zip(*got))


def _inside(v, R):
    a, b = R, np.roll(R, -1, 0)
    m = (a[:, 1] > v[1]) != (b[:, 1] > v[1])
    a, b = a[m], b[m]
    return bool((v[0] < a[:, 0] + (v[1] - a[:, 1]) / (b[:, 1] - a[:, 1]) * (b[:, 0] - a[:, 0])).sum() & 1)


def _clip(P, Q, union):
    """The rings of P clipped with Q in general position (Greiner and Hormann 1998), from the
    first crossing along P on; None where they neither cross nor contain each other."""
    p, q, a, b = _crossings(P, Q)
    n = len(p)
    if n == 0:
        in_p, in_q = _inside(P[0], Q), _inside(Q[0], P)
        return None if not (in_p or in_q) else [R for R, i in ((P, in_p), (Q, in_q)) if i != union]
    X = (1.0 - a)[:, None] * P[p] + a[:, None] * np.roll(P, -1, 0)[p]
    rings, at, entry = [], [], []
    for V, W, e, t in ((P, Q, p, a), (Q, P, q, b)):
        order = np.lexsort((t, e))
        slot = np.empty(n, np.int64)
        slot[order] = e[order] + 1 + np.arange(n)
        xy = np.empty((len(V) + n, 2))
        mask = np.ones(len(xy), bool)
        mask[slot] = False
        xy[mask], xy[slot] = V, X
        flag = np.zeros(len(xy), np.int8)                   # 1 entry, 2 exit, from the first vertex on
        out = not _inside(V[0], W)
        flag[slot[order]] = np.where((np.arange(n) % 2 == 0) == out, 1, 2)
        rings.append(xy)
        at.append(slot)
        entry.append(flag)
    twin = [dict(zip(at[0], at[1])), dict(zip(at[1], at[0]))]
    seen, comps = set(), []
    for start in np.sort(at[0]):
        if start in seen:
            continue
        side, v, comp = 0, start, []
        while True:
            seen.add(v if side == 0 else twin[1][v])
            step = 1 if (entry[side][v] == 1) != union else -1
            while True:
                v = (v + step) % len(rings[side])
                comp.append(rings[side][v])
                if entry[side][v]:
                    break
            seen.add(v if side == 0 else twin[1][v])
            if side == 0 and v == start:
                break
            v, side = twin[side][v], 1 - side
            if side == 0 and v == start:
                break
        comps.append(np.array(comp))
    return comps


def _tidy(c, eps=1e-7):
    """A ring without the vertices that lie on a line with their neighbours, in one pass."""
    if not (np.abs(_side(np.roll(c, 1, 0), c, np.roll(c, -1, 0))) < eps).any():
        return c
    r = 0
    while r < len(c) and (r == len(c) - 1 or abs(_side(c[-1], c[r], c[r + 1])) < eps):
        r += 1
    kept = [v for v in c[r:r + 1]]
    for j in range(r + 1, len(c)):
        if abs(_side(kept[-1], c[j], c[j + 1] if j + 1 < len(c) else c[r])) >= eps:
            kept.append(c[j])
    return np.array(kept).reshape(-1, 2)


def _pair_xy(P, Q, union=False):
    comps = _clip(P, Q, union)
    return None if comps is None else np.concatenate([_tidy(c).reshape(-1) for c in comps] or [np.zeros(0)])


def _laid_out(case, name, values):
    """run()'s buffers with `values` at the front of one of them, nothing for the others."""
    sizes = _capacity(case)
    out = dict.fromkeys(sizes)
    out[name] = np.zeros(sizes[name])
    if values is not None:
        out[name][:len(values)] = values
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "pair" and case["np"] * case["nq"] <= 30_000_000:
        P, Q = (r.reshape(-1, 2) for r in _pair_rings(case, seed))
        return _laid_out(case, "xy", _pair_xy(P, Q))
    if kind not in ("join", "mbr") or (kind == "join" and max(case["nb"], case["no"]) > 4000):
        return None
    layers, boxes = _layers(case, seed), []
    for xy, vnum, vps in layers:
        pid = torch.repeat_interleave(torch.arange(vnum.numel(), device=_DEV), vnum.long())
        box = [torch.full((vnum.numel(),), v, dtype=torch.float64, device=_DEV) for v in (math.inf, math.inf, -math.inf, -math.inf)]
        for i in range(4):
            box[i].scatter_reduce_(0, pid, xy[i % 2::2].contiguous(), "amin" if i < 2 else "amax")
        boxes.append(torch.stack(box, 1))
    B, O = boxes
    found = []
    step = max(1, 200_000_000 // O.shape[0])
    for i in range(0, B.shape[0], step):                    # every overlapping pair of boxes, by (base, overlay)
        b = B[i:i + step, None]
        hit = (b[..., 0] <= O[None, :, 2]) & (O[None, :, 0] <= b[..., 2]) & (b[..., 1] <= O[None, :, 3]) & (O[None, :, 1] <= b[..., 3])
        found.append(hit.nonzero() + torch.tensor([i, 0], device=_DEV))
        del hit
    bo = torch.cat(found)
    if kind == "mbr":
        b, o = B[bo[:, 0]], O[bo[:, 1]]
        cmbr = torch.cat([torch.maximum(b[:, :2], o[:, :2]), torch.minimum(b[:, 2:], o[:, 2:])], 1)
        return _laid_out(case, "cmbr", cmbr.reshape(-1).cpu().numpy())
    host = [synth.Layer(xy.cpu().numpy(), vnum.cpu().numpy()) for xy, vnum, _ in layers]
    parts = []
    for b, o in bo.cpu().tolist():
        P, Q = host[0].ring(b), host[1].ring(o)
        xy = _pair_xy(*((Q, P) if len(P) < len(Q) else (P, Q)), case["union"])   # the longer ring is clipped
        if xy is not None:
            parts.append(xy)
    return _laid_out(case, "xy", np.concatenate(parts or [np.zeros(0)]))
