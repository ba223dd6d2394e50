"""Workloads for timing this library, each through a public entry point.

A case is a dict of plain values:

* ``kind``     the entry point: ``event`` (``Context.cluster_event``, one event per
               call), ``batch`` (``Context.cluster_batch_device``), ``graph`` (a
               captured batch call and the jet epilogue ``Context.select_jets``),
               ``host`` (``Context.cluster_batch``, host arrays in and out) or
               ``server`` (``Server.submit`` / ``Server.poll``);
* ``events``   events per call, with particle counts log-uniform in [``lo``, ``hi``]
               (with ``serve``: the serving mix's lognormal counts clipped to it);
* ``algo``, ``radius``  the algorithm (1 kt, 0 C/A, -1 anti-kt) and R; with ``serve``
               they are per event, as the serving mix has them (70 % anti-kt R=0.4,
               15 % kt R=0.6, 15 % C/A R=0.8);
* ``shape``    ``hard`` (jets over a soft background, |eta| < 5) or ``pileup`` (dense
               soft background, |eta| < 4, 2-6 hard axes);
* ``history``  the merge history and the constituents' jets are returned too.

Inputs come from ``fastjet_gpu_gb300.events``, the generators that the tests and
the benchmark use.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fastjet_gpu_gb300 as F
from fastjet_gpu_gb300 import events as ev


def listed():
    return [
        # one event per call, as the reference's driver does: a handful of
        # particles (a quiet collision), where the launches are most of the call
        case("event-50", "event", 1, 50, 50, -1, 0.4),
        # an ordinary event of the size of the reference's 354-particle fixture,
        # with its merge history (substructure studies use wide kt jets)
        case("event-354-kt-history", "event", 1, 354, 354, 1, 1.0, history=True),
        # the top of the mixed workload, alone: the latency of one request
        case("event-2000", "event", 1, 2000, 2000, -1, 0.4),
        # a trigger-like batch of small events of odd sizes
        case("batch-96-small", "batch", 96, 17, 301, -1, 0.4),
        # Cambridge/Aachen fat jets of a medium batch, with the history that
        # declustering reads
        case("batch-400-cam-history", "batch", 400, 50, 4000, 0, 0.8, history=True),
        # the benchmark's batch: 4096 events of 50-2000 particles
        case("batch-4096", "batch", 4096, 50, 2000, -1, 0.4),
        # repeated batches through a captured graph, jets filtered and sorted
        case("graph-1024-kt", "graph", 1024, 50, 2000, 1, 0.6),
        # host arrays in and out, per-event algorithm and R, up to 20k particles
        case("host-256-serve", "host", 256, 100, 20000, serve=True, history=True),
        # a burst of requests to the server
        case("server-192", "server", 192, 100, 4000, serve=True),
        # one pile-up event per call
        case("event-12001-pileup", "event", 1, 12001, 12001, -1, 0.4, shape="pileup"),
        # the benchmark's pile-up workload: 64 events of 10k-60k particles
        case("batch-64-pileup", "batch", 64, 10000, 60000, -1, 0.4, shape="pileup"),
        # pile-up with kt (its areas set the pile-up density), smaller events
        case("batch-40-pileup-kt", "batch", 40, 5000, 30000, 1, 0.6, shape="pileup"),
    ]


def case(name, kind, events, lo, hi, algo=-1, radius=0.4, shape="hard", serve=False, history=False):
    return {"name": name, "kind": kind, "events": events, "lo": lo, "hi": hi, "algo": algo, "radius": radius,
            "shape": shape, "serve": serve, "history": history}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["event", "event", "batch", "batch", "graph", "host", "server", "pileup"])
    algo = rng.choice([-1, -1, 0, 1])
    radius = rng.choice([0.3, 0.4, 0.5, 0.6, 0.8, 1.0])
    history = rng.random() < 0.4
    if kind == "event":
        n = _log_int(rng, 30, 4096)
        c = case("", "event", 1, n, n, algo, radius, history=history)
    elif kind == "pileup":
        lo = _log_int(rng, 4097, 20000)
        n = _log_int(rng, 1, 24)
        c = case("", "event" if n == 1 else "batch", n, lo, lo if n == 1 else 2 * lo + 1, algo,
                 min(radius, 0.6), shape="pileup", history=history)
    elif kind == "server":
        c = case("", "server", _log_int(rng, 16, 256), 100, _log_int(rng, 500, 6000), serve=True, history=history)
    elif kind == "host":
        c = case("", "host", _log_int(rng, 4, 512), 100, _log_int(rng, 1000, 20000), serve=True, history=history)
    else:
        lo = _log_int(rng, 20, 400)
        c = case("", kind, _log_int(rng, 16, 3000), lo, _log_int(rng, lo + 50, 2500), algo, radius, history=history)
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs

def _sizes(case):
    """The events' particle counts: a fixed spread over the case's range, so that
    the buffers of two inputs of a case have the same shapes."""
    rng = np.random.default_rng([case["events"], case["lo"], case["hi"]])
    if case["serve"]:  # the serving mix: lognormal, median 1500, sigma 0.8
        x = rng.normal(math.log(1500.0), 0.8, case["events"])
    else:
        x = rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["events"])
    return np.clip(np.rint(np.exp(x)), case["lo"], case["hi"]).astype(np.int64)


def _inputs(case, seed):
    """(Batch, per-event algorithms or a scalar, per-event R or a scalar)."""
    sizes = _sizes(case)
    rng = np.random.default_rng(seed)
    algo, radius = case["algo"], case["radius"]
    if case["serve"]:
        u = rng.random(sizes.size)
        algo = np.where(u < 0.70, -1, np.where(u < 0.85, 1, 0)).astype(np.int32)
        radius = np.where(u < 0.70, 0.4, np.where(u < 0.85, 0.6, 0.8))
    pileup = case["shape"] == "pileup"
    axes = rng.integers(2, 7, sizes.size) if pileup else rng.poisson(3, sizes.size) + 1
    seeds = rng.integers(0, 2**62, sizes.size)
    soft = {"soft_mean": 0.6, "soft_eta": 4.0} if pileup else {}
    evs = [ev.single_event(int(n), int(a), int(s), **soft) for n, a, s in zip(sizes, axes, seeds)]
    offsets = np.zeros(sizes.size + 1, np.int64)
    np.cumsum(sizes, out=offsets[1:])
    return ev.Batch(np.concatenate(evs), offsets), algo, radius


def _device_outputs(total, n_events, history):
    """Output buffers a program keeps; zeroed, as only the jets' rows are written."""
    out = {"jets": torch.zeros((total, 4), dtype=torch.float64, device="cuda"),
           "jet_label": torch.zeros(total, dtype=torch.int32, device="cuda"),
           "n_jets": torch.zeros(n_events, dtype=torch.int32, device="cuda")}
    if history:
        out["history"] = torch.zeros((total, 2), dtype=torch.float64, device="cuda")
        out["owner"] = torch.zeros(total, dtype=torch.int32, device="cuda")
    return out


def prepare(case, seed):
    ctx = F.default_context(0)
    batch, algo, radius = _inputs(case, seed)
    s = {"case": case, "ctx": ctx, "algo": algo, "radius": radius}
    kind = case["kind"]
    if kind in ("host", "server"):
        s["particles"], s["offsets"] = batch.particles, batch.offsets
        if kind == "server":
            s["server"] = F.Server(ctx, arena_particles=1 << 20, history=case["history"])
        return s
    s["p4"] = torch.from_numpy(batch.particles).cuda()
    if kind == "event":
        s["row"] = torch.arange(batch.particles.shape[0], device="cuda")
        return s
    s["offsets"] = torch.from_numpy(batch.offsets).cuda()
    s["out"] = _device_outputs(batch.particles.shape[0], batch.n_events, case["history"])
    if kind == "graph":
        s["graph"] = ctx.capture_batch(s["p4"], s["offsets"], algo, radius, history=case["history"],
                                       owner=case["history"], out=s["out"])
    return s


# --------------------------------------------------------------------- runs

def _history(out):
    """The history's labels and distances, and the constituents' jets."""
    h = out.get("history")
    if h is None:
        return {}
    if isinstance(h, torch.Tensor):
        return {"step": h.view(torch.int32)[:, :2], "d": h[:, 1], "owner": out["owner"]}
    return {"step": np.stack([h["a"], h["b"]], 1), "d": h["d"], "owner": out["owner"]}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind, history = case["kind"], case["history"]
    if kind == "event":
        out = ctx.cluster_event(state["p4"], case["algo"], case["radius"], history=history, owner=history)
        # rows past the jet count are not written: fixed-shape programs mask them
        live = state["row"] < out["n_jets"]
        return {"jets": torch.where(live[:, None], out["jets"], 0.0),
                "jet_label": torch.where(live, out["jet_label"], 0), "n_jets": out["n_jets"], **_history(out)}
    if kind == "batch":
        out = ctx.cluster_batch_device(state["p4"], state["offsets"], case["algo"], case["radius"],
                                       history=history, owner=history, out=state["out"])
        return {"jets": out["jets"], "jet_label": out["jet_label"], "n_jets": out["n_jets"], **_history(out)}
    if kind == "graph":
        state["graph"].launch()
        out = state["out"]
        hard = ctx.select_jets(out, state["offsets"], ptmin=5.0)
        return {"n_hard": hard["n_jets"], "jets": out["jets"], "jet_label": out["jet_label"],
                "n_jets": out["n_jets"], **_history(out)}
    off = state["offsets"]
    if kind == "host":
        out = ctx.cluster_batch(state["particles"], off, state["algo"], state["radius"],
                                history=history, owner=history)
        first = np.repeat(off[:-1], np.diff(off))
        live = np.arange(off[-1]) - first < np.repeat(out["n_jets"], np.diff(off))
        return {"jets": np.where(live[:, None], out["jets"], 0.0), "jet_label": np.where(live, out["jet_label"], 0),
                "n_jets": out["n_jets"], **_history(out)}
    srv = state["server"]
    event_of = {}
    for e in range(off.size - 1):
        t = srv.submit(state["particles"][off[e]:off[e + 1]], int(state["algo"][e]), float(state["radius"][e]))
        event_of[t] = e
    total = int(off[-1])
    out = {"jets": np.zeros((total, 4)), "jet_label": np.zeros(total, np.int32),
           "n_jets": np.zeros(off.size - 1, np.int32)}
    if history:
        out.update(history=np.zeros(total, F.STEP), owner=np.zeros(total, np.int32))
    left = off.size - 1
    while left:
        for d in srv.poll(64, timeout_us=2000):
            e = event_of[d["ticket"]]
            o, k = off[e], d["n_jets"]
            out["jets"][o:o + k], out["jet_label"][o:o + k], out["n_jets"][e] = d["jets"], d["jet_label"], k
            if history:
                out["history"][o:off[e + 1]], out["owner"][o:off[e + 1]] = d["history"], d["owner"]
            left -= 1
    return {"jets": out["jets"], "jet_label": out["jet_label"], "n_jets": out["n_jets"], **_history(out)}


def work(case):
    """Momenta in; jets (about one row per seven particles in these events),
    counts, history and owners out.  The merges' arithmetic depends on the
    event, so only the bytes are stated."""
    n = int(_sizes(case).sum())
    return {"bytes": n * (32 + 36 / 7 + (20 if case["history"] else 0)) + 12 * case["events"], "flops": 0}


# -------------------------------------------------------------------- exact

def _cluster_exact(p4, algo, radius):
    """Generalised-kt clustering of one event in plain numpy, E-scheme, every
    distance recomputed for the pseudojet that a step makes."""
    n = p4.shape[0]
    p = p4.copy()
    inv_r2 = 1.0 / (radius * radius)

    def kin(v):
        pt2 = v[..., 0] ** 2 + v[..., 1] ** 2
        phi = np.arctan2(v[..., 1], v[..., 0]) % (2 * math.pi)
        m2 = np.maximum(0.0, (v[..., 3] + v[..., 2]) * (v[..., 3] - v[..., 2]) - pt2)
        epz = v[..., 3] + np.abs(v[..., 2])
        rap = 0.5 * np.log((pt2 + m2) / (epz * epz))
        w = pt2 if algo == 1 else np.ones_like(pt2) if algo == 0 else 1.0 / pt2
        return np.where(v[..., 2] > 0, -rap, rap), phi, w

    rap, phi, w = (np.array(x) for x in kin(p))

    def dist(s):  # dR2 to slot s, of every slot alive
        dphi = np.abs(phi - phi[s])
        dphi = np.where(dphi > math.pi, 2 * math.pi - dphi, dphi)
        d = dphi * dphi + (rap - rap[s]) ** 2
        d[~alive] = np.inf
        d[s] = np.inf
        return d

    alive = np.ones(n, bool)
    nn, nd = np.zeros(n, np.int64), np.zeros(n)
    for s in range(n):
        d = dist(s)
        nn[s] = np.argmin(d)
        nd[s] = d[nn[s]]
    owner = np.arange(n)
    jets, labels, steps, ds = [], [], [], []
    for _ in range(n):
        key = np.minimum(np.where(np.isfinite(nd), np.minimum(w, w[nn]) * nd * inv_r2, np.inf), w)
        key[~alive] = np.inf
        c = int(np.argmin(key))
        if key[c] < w[c]:
            a, b = min(c, int(nn[c])), max(c, int(nn[c]))
            steps.append((a, b))
            ds.append(key[c])
            p[a] += p[b]
            owner[owner == b] = a
            rap[a], phi[a], w[a] = kin(p[a])
        else:
            a, b = -1, c
            steps.append((c, -1))
            ds.append(w[c])
            jets.append(p[c].copy())
            labels.append(c)
        alive[b] = False
        nd[b] = np.inf
        if a >= 0:
            d = dist(a)
            closer = alive & (d < nd)
            nd[closer], nn[closer] = d[closer], a
            nn[a] = np.argmin(d)
            nd[a] = d[nn[a]]
        for t in np.nonzero(alive & ((nn == b) | (nn == a)))[0]:
            d = dist(t)
            nn[t] = np.argmin(d)
            nd[t] = d[nn[t]]
    jet_of = np.zeros(n, np.int64)
    jet_of[labels] = np.arange(len(labels))
    return np.array(jets).reshape(-1, 4), labels, steps, ds, jet_of[owner]


def exact(case, seed):
    if case["kind"] not in ("event", "batch") or case["events"] * case["hi"] > 40000 or case["hi"] > 2500:
        return None
    batch, algo, radius = _inputs(case, seed)
    total, off = batch.particles.shape[0], batch.offsets
    out = {"jets": np.zeros((total, 4)), "jet_label": np.zeros(total, np.int32),
           "n_jets": np.zeros(batch.n_events, np.int32), "step": np.zeros((total, 2), np.int32),
           "d": np.zeros(total), "owner": np.zeros(total, np.int32)}
    for e in range(batch.n_events):
        o = off[e]
        jets, labels, steps, ds, owner = _cluster_exact(batch.event(e), algo, radius)
        k = len(labels)
        out["jets"][o:o + k], out["jet_label"][o:o + k], out["n_jets"][e] = jets, labels, k
        out["step"][o:off[e + 1]], out["d"][o:off[e + 1]], out["owner"][o:off[e + 1]] = steps, ds, owner
    if not case["history"]:
        for k in ("step", "d", "owner"):
            del out[k]
    return out
