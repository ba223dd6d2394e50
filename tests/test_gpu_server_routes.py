"""Request server: micro-batches for the rounds kernel and for the step-by-step
kernels beside each other, in every size bucket: each result is that of the same
event clustered alone."""
import numpy as np
import pytest

from fastjet_gpu_gb300 import events as E
from test_gpu_server import _drive, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fastjet_gpu_gb300 as F
    c = F.Context(0)
    yield c
    c.close()


# (one stream: queued requests go out many at a time; a request with the GPU to itself has a rule of its own)
@pytest.mark.parametrize("streams,max_batch", [(1, 64), (2, 3), (16, 512)])
def test_routes_of_every_bucket(ctx, streams, max_batch):
    import fastjet_gpu_gb300 as F
    rng = np.random.default_rng(streams)
    sizes = [90, 112, 250, 300, 513, 600, 1000, 1025, 2000, 2049, 3000, 4097] * 5
    events, algo, radius = [], [], []
    for i, n in enumerate(sizes):
        ev = E.single_event(n, 1 + i % 4, 7000 + i)
        if i % 7 == 0:
            ev[n // 2, :2] = 0.0  # kt: left to the step-by-step kernels
        events.append(ev)
        a, r = [(-1, 0.4), (1, 0.6), (-1, 1.2), (0, 0.8), (1, 2.5)][int(rng.integers(0, 5))]
        algo.append(a)
        radius.append(r)
    srv = F.Server(ctx, history=True, streams=streams, max_batch=max_batch)
    try:
        res = _drive(srv, events, np.array(algo, np.int32), np.array(radius), per_poll=50, seed=streams)
    finally:
        srv.close()
    for e, ev in enumerate(events):
        _same(ctx, res[e], ev, algo[e], radius[e], f"request {e} of {ev.shape[0]}")
