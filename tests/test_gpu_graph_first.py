"""A capture as the first thing that a process does: whatever the launches ask of the
runtime (attributes, occupancies) is asked before the capture begins."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
import numpy as np, torch
import fastjet_gpu_gb300 as F
import gpu_util as U
from fastjet_gpu_gb300 import events as E
count, radius = int(sys.argv[1]), float(sys.argv[2])
sizes = [60, 300, 700, 1500, 2100, 4500, 330][:count] + [40] * max(0, count - 7)
b = E._batch_from([E.single_event(n, 3, seed=n) for n in sizes])
ctx = F.Context(0)
g = ctx.capture_batch(torch.from_numpy(b.particles).cuda(), torch.from_numpy(b.offsets).cuda(), -1, radius,
                      history=True, owner=True)
g.launch()
g.check()
out = {k: v.cpu().numpy() for k, v in g.out.items() if k != "history"}
out["history"] = F.history_records(g.out["history"])
for e in range(min(count, 8)):
    s = slice(b.offsets[e], b.offsets[e + 1])
    U.compare_event(b.event(e), -1, radius, out["jets"][s], out["n_jets"][e], out["history"][s], out["owner"][s],
                    out["jet_label"][s], f"event {e}")
print("ok")
"""


# up to an SM per event, up to half of one, and more; step by step and with rounds
@pytest.mark.parametrize("count,radius", [(1, 1.2), (7, 1.2), (7, 0.4), (200, 1.2), (200, 0.4), (400, 0.4)])
def test_capture_before_anything_else(count, radius):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.path.join(ROOT, "tests"))
    res = subprocess.run([sys.executable, "-c", PROGRAM, str(count), str(radius)], env=env, cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and res.stdout.endswith("ok\n"), res.stdout[-2000:] + res.stderr[-4000:]
