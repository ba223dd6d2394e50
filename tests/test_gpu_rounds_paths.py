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


def _main(groups):
    import torch

    import fastjet_gpu_gb300 as F
    import gpu_util as U
    from fastjet_gpu_gb300 import events as E
    ctx = F.Context(0)
    out = []
    for g in groups:
        rows = []
        for i in g["which"]:
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
