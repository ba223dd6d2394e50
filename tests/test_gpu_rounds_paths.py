"""The rounds kernel's rarer ways (csrc/fjg_cluster_rounds.cuh), seen through the
phase-counter build: that the inputs meant for a way do take it, and that the
results are the oracle's bit for bit all the same.

The counters need another library in the process, so each test runs this file as a
program in a process of its own, which prints the counters of each event.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
DENSE = {"soft_mean": 0.6, "soft_eta": 4.0}

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def counters():
    """counters(groups) -> the counters of each event, alone, of each group."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from fastjet_gpu_gb300 import build as B
    lib = B.build(phase_clocks=True)

    def run(groups):
        env = dict(os.environ, FJG_LIB=lib, PYTHONPATH=ROOT + os.pathsep + HERE)
        res = subprocess.run([sys.executable, os.path.abspath(__file__), json.dumps(groups)], env=env, cwd=ROOT,
                             capture_output=True, text=True, timeout=600)
        assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
        return json.loads(res.stdout.splitlines()[-1])

    return run


def _total(events, key):
    return sum(e[key] for e in events)


def test_steps_taken_back(counters):
    """Two hard jets near each other, whose lines of steps the rounds run side by
    side, in the order of one after the other: the later one is taken back.  Slots
    in shared memory and in the workspace."""
    small, r04, r06, r10 = counters([
        {"n": 1500, "radius": 0.8, "which": list(range(18, 26))},
        {"n": 10000, "radius": 0.4, "which": [4, 19, 23, 26, 38], "dense": True},
        {"n": 10000, "radius": 0.6, "which": [6, 10, 11, 18, 22, 23, 34, 36], "dense": True},
        {"n": 6000, "radius": 1.0, "which": [10, 23, 31], "dense": True}])
    for group in (small, r04, r06, r10):
        assert _total(group, "r_undone") > 0 and _total(group, "r_conflict_d") > 0
        assert _total(group, "r_retries") == 0 and _total(group, "r_events") == len(group)
    # a line that came too early goes back as a whole: no event does its rounds twice over
    for e in r04 + r06 + r10:
        assert e["r_undone"] < e["r_rounds"] / 2, e


# (one event; an SM each; an SM for two; many)
@pytest.mark.parametrize("count", [1, 60, 200, 330])
def test_events_left_to_the_other_kernels(counters, count):
    """Particles without pT (kt), and particles on a lattice (ties): events that the
    rounds hand on, from every list, beside events that they keep."""
    sizes = [5000, 4097, 4000, 2100, 2048, 1500, 1025, 1024, 700, 600, 513, 512, 450] * 20 + [256, 200, 100] * 24
    sizes = sizes[:count - 3] + [700, 2049, 300] if count > 1 else [700]
    batch, = counters([{"sizes": sizes, "algo": 1, "radius": 0.6, "kinds": ["no pT", "lattice", "jets"]}])
    row, = batch
    assert row["r_retries"] > 0
    assert row["r_events"] > 0 or count == 1
    # every event is clustered by one kernel, and only what that one hands on by a second
    assert row["events"] + row["t_events"] + row["r_events"] == count
    assert row["events"] + row["t_events"] >= row["r_retries"]


def test_lattice_is_left_at_once(counters):
    """Neighbours at the same distance by the hundred: no round is tried."""
    for algo, radius in ((-1, 0.4), (0, 0.8)):
        batch, = counters([{"sizes": [700, 1024, 1500, 3000, 5000], "algo": algo, "radius": radius,
                            "kinds": ["lattice"]}])
        row, = batch
        assert row["r_retries"] == 5 and row["events"] + row["t_events"] == 5
        assert row["r_conflict_a"] + row["r_conflict_b"] + row["r_conflict_d"] + row["r_events"] == 0


def _particles(kind, n, i):
    from fastjet_gpu_gb300 import events as E
    if kind == "lattice":
        r = np.random.default_rng(i)
        y, phi, pt = r.integers(-30, 31, n) * 0.125, r.integers(0, 50, n) * 0.125, r.integers(1, 8, n) * 0.5
        return np.stack([pt * np.cos(phi), pt * np.sin(phi), pt * np.sinh(y), pt * np.cosh(y)], 1)
    p4 = E.single_event(n, 1 + i % 5, 5000 * n + i)
    if kind == "no pT":
        p4[n // 2, :2] = 0.0
    return p4


def _batch(ctx, g):
    import gpu_util as U
    evs = [_particles(g["kinds"][i % len(g["kinds"])], n, i) for i, n in enumerate(g["sizes"])]
    off = np.concatenate([[0], np.cumsum(g["sizes"])]).astype(np.int64)
    ctx.phase_clocks(reset=True)
    res = ctx.cluster_batch(np.concatenate(evs), off, g["algo"], g["radius"], history=True, owner=True)
    counts = ctx.phase_clocks()
    for e, p4 in enumerate(evs):
        s = slice(off[e], off[e + 1])
        U.compare_event(p4, g["algo"], g["radius"], res["jets"][s], res["n_jets"][e], res["history"][s],
                        res["owner"][s], res["jet_label"][s], f"event {e} of {len(p4)}")
    return counts


def _main(groups):
    import torch

    import fastjet_gpu_gb300 as F
    import gpu_util as U
    from fastjet_gpu_gb300 import events as E
    ctx = F.Context(0)
    out = []
    for g in groups:
        rows = []
        if "sizes" in g:
            rows.append(_batch(ctx, g))
        for i in g.get("which", []):
            n = g["n"]
            p4 = E.single_event(n, 1 + i % 5, 5000 * n + i, **(DENSE if g.get("dense") else {}))
            ctx.phase_clocks(reset=True)
            res = ctx.cluster_event(torch.from_numpy(p4).cuda(), g.get("algo", -1), g["radius"], history=True,
                                    owner=True)
            rows.append(ctx.phase_clocks())
            U.compare_event(p4, g.get("algo", -1), g["radius"], res["jets"].cpu().numpy(), int(res["n_jets"][0]),
                            F.history_records(res["history"]), res["owner"].cpu().numpy(),
                            res["jet_label"].cpu().numpy(), f"n {n} R {g['radius']} event {i}")
        out.append(rows)
    print(json.dumps(out))


if __name__ == "__main__":
    _main(json.loads(sys.argv[1]))
