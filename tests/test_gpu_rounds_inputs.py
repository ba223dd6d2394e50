"""The rounds kernel (csrc/fjg_cluster_rounds.cuh) on inputs at the ends of the
number range, against the CPU oracle bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

import fastjet_gpu_gb300 as F  # noqa: E402
import gpu_util as U  # noqa: E402
from fastjet_gpu_gb300 import events as E  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    return F.Context(0)


def _check_event(ctx, p4, algo, radius, tag):
    out = ctx.cluster_event(torch.from_numpy(p4).cuda(), algo, radius, history=True, owner=True)
    U.compare_event(p4, algo, radius, out["jets"].cpu().numpy(), int(out["n_jets"][0]),
                    F.history_records(out["history"]), out["owner"].cpu().numpy(),
                    out["jet_label"].cpu().numpy(), tag)


def _on_the_beam(pz):
    """Particles without pT and mass: their rapidity is 1e5 + |pz|."""
    pz = np.asarray(pz, np.float64)
    return np.stack([0 * pz, 0 * pz, pz, np.abs(pz)], 1)


# the smallest event alone that the kernel takes, slots in shared memory and in the workspace
@pytest.mark.parametrize("n", [224, 600, 4200])
def test_particles_on_the_beam_line(ctx, n):
    """Rapidities of 1e5, where FP32 coordinates are 2^-7 apart: particles just
    within R of one another, whose weights are all the same 1e300."""
    base = E.single_event(n, 3, 91 + n)
    rng = np.random.default_rng(n)
    chains = [[10.8019, 10.4024, 10.0038]]
    chains += [rng.uniform(1, 50) + np.cumsum(rng.uniform(0.37, 0.402, 7)) * rng.choice([-1, 1]) for _ in range(6)]
    for i, pz in enumerate(chains):
        pz = np.asarray(pz) * (1 if i % 2 == 0 else -1)
        for algo in (-1, 0, 1):
            _check_event(ctx, np.concatenate([_on_the_beam(pz), base]), algo, 0.4, f"n {n} chain {i} algo {algo}")


# (alone: the rounds kernel's sizes, which hands such an event on; 100 and R = 3: the step-by-step kernels at once)
@pytest.mark.parametrize("n,radius", [(100, 0.4), (300, 0.4), (1500, 3.0), (4200, 0.4), (4200, 3.0)])
def test_infinite_rapidity(ctx, n, radius):
    """No pT and E below |pz| (rounded input): the rapidity is infinite, and so is
    the distance to everything; two of them are a NaN apart.  Every neighbour
    search has to find some slot all the same."""
    p4 = E.single_event(n, 3, 17 + n)
    beam = _on_the_beam([20.0, 30.0, -7.0, -8.0, 3.0])
    beam[:, 3] *= 1.0 - 2.0 ** -40
    for at in (0, n // 2, n):
        p = np.concatenate([p4[:at], beam, p4[at:]])
        for algo in (-1, 0):
            _check_event(ctx, p, algo, radius, f"n {n} R {radius} at {at} algo {algo}")


def test_sums_that_overflow(ctx):
    """A merged jet's pT^2 or E that is beyond the number range: its rapidity is
    infinite or NaN.  Such an event gives some result or an error, and the next
    one is clustered as ever."""
    base = E.single_event(400, 3, 23)
    for scale in (1e153, 1e154, 1e200):
        for algo in (-1, 0, 1):
            try:
                out = ctx.cluster_event(torch.from_numpy(base * scale).cuda(), algo, 0.4)
                assert 0 <= int(out["n_jets"][0]) <= base.shape[0]
            except F.FjgError:
                pass
    _check_event(ctx, base, -1, 0.4, "after")


def test_no_workspace_where_the_rounds_take_nothing():
    """The rounds kernel's workspace (480 bytes a particle) is not allocated for calls
    that its rule refuses; with it, the results are the same as without."""
    ctx = F.Context(0)
    evs = [E.single_event(600, 3, i) for i in range(8)]
    p4 = torch.from_numpy(np.concatenate(evs * 250)).cuda()
    off = torch.arange(0, 600 * 2000 + 1, 600, dtype=torch.int64, device="cuda")
    out = ctx.cluster_batch_device(p4, off, -1, 0.4, out=None)
    torch.cuda.synchronize()
    ctx.close()
    ctx = F.Context(0)
    free = [torch.cuda.mem_get_info()[0]]
    for radius in (1.2, 0.4):
        ctx.cluster_batch_device(p4, off, -1, radius, out=out)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    n = p4.shape[0]
    assert free[0] - free[1] < 300 * n  # the other workspaces: 70 + 120 bytes a particle
    assert free[1] - free[2] > 384 * n
    ctx.close()
