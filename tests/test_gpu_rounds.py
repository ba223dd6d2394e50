"""The rounds kernel (csrc/fjg_cluster_rounds.cuh) against the CPU oracle, at the
sizes where its dispatch, its shared-memory layouts and its tile grids change.

Every comparison is bit for bit (history, distances, jets, constituents), as in
the other parity tests: the kernel takes steps out of order and sorts them, so a
step in the wrong place shows in the history.
"""
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


# lists of 256 << b particles, the smallest events the kernel takes alone (224, kt
# and C/A 200) or among some (112), the end of the shared-memory slots (4096), an odd size above it
SIZES = [111, 112, 199, 200, 223, 224, 255, 257, 512, 513, 1023, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 6001]


@pytest.mark.parametrize("n", SIZES)
def test_sizes(ctx, n):
    for algo, radius in ((-1, 0.4), (1, 0.6), (0, 0.8)):
        _check_event(ctx, E.single_event(n, 3, 31 * n + algo), algo, radius, f"n {n} algo {algo}")


# radii: one tile or few (3.0: refused by the rule, 1.5 and 1.05 at its edge),
# more tiles than there is room for (0.02), none at all (0)
@pytest.mark.parametrize("radius", [0.0, 0.02, 0.1, 0.85, 1.05, 1.5, 3.0])
def test_radii(ctx, radius):
    for algo in (-1, 0, 1):
        _check_event(ctx, E.single_event(600, 4, 77), algo, radius, f"R {radius} algo {algo}")


def test_dense_and_wide_range(ctx):
    """Dense lists (many slots a tile) and the size from which anti-kt events
    begin with the wider range."""
    ev = E.portable_pileup([20001, 9000])
    _check_event(ctx, ev[0], -1, 0.4, "20001 anti-kt")
    _check_event(ctx, ev[1], 1, 0.6, "9000 kt")


def test_ties_go_to_the_step_by_step_kernels(ctx):
    """Exact ties, weightless particles and a slot that hundreds of others are
    nearest to: conflicts by design, clustered by the other kernels."""
    base = E.single_event(500, 3, 5)
    mirrored = base.copy()
    mirrored[:, 2] *= -1.0  # the same distances at the opposite rapidity
    zero = base.copy()
    zero[::25, :2] = 0.0
    cases = {"mirrored": np.concatenate([base, mirrored]), "repeated": np.concatenate([base, base[:150]]),
             "one repeated": np.concatenate([base, np.repeat(base[:1], 300, axis=0)]), "no pT": zero,
             "all the same": np.repeat(base[:1], 300, axis=0)}
    for name, p4 in cases.items():
        for algo in (-1, 0, 1):
            _check_event(ctx, np.ascontiguousarray(p4), algo, 0.4, f"{name} algo {algo}")


@pytest.mark.parametrize("count", [40, 200, 320])
def test_many_events_mixed_rules(ctx, count):
    """Events that have an SM each, that share one by two, and more: a rule each,
    per event (algorithm and R from arrays), both kernels on one list; and the same
    batch through a captured graph."""
    sizes = [5000, 3000, 2100, 1500, 1100, 900, 700, 600, 513, 512, 450, 400, 399] + [20 + i % 60 for i in range(307)]
    sizes = sizes[:count - 8] + [250, 230, 210, 200, 190, 150, 113, 100]
    evs = [E.single_event(n, 1 + i % 4, 900 + i) for i, n in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    p4 = np.ascontiguousarray(np.concatenate(evs))
    algo = np.array([(-1, 1, 0)[i % 3] for i in range(len(sizes))], np.int32)
    radius = np.array([(0.4, 0.6, 0.8, 1.0)[(i // 3) % 4] for i in range(len(sizes))])
    res = ctx.cluster_batch(p4, off, algo, radius, history=True, owner=True)
    for e in range(len(sizes)):
        s = slice(off[e], off[e + 1])
        U.compare_event(p4[s], int(algo[e]), float(radius[e]), res["jets"][s], res["n_jets"][e], res["history"][s],
                        res["owner"][s], res["jet_label"][s], f"event {e}")
    g = ctx.capture_batch(torch.from_numpy(p4).cuda(), torch.from_numpy(off).cuda(), torch.from_numpy(algo).cuda(),
                          torch.from_numpy(radius).cuda(), history=True, owner=True)
    for _ in range(2):
        g.launch()
        g.check()
    out = {k: v.cpu().numpy() for k, v in g.out.items() if k != "history"}
    out["history"] = F.history_records(g.out["history"])
    U.same_results(out, res, off)


def test_steps_taken_back(ctx):
    """Events in which a step is found to have come too early (dense, R = 0.6 and
    0.8; above 4096 particles the slots' state is in the workspace): the steps
    since are taken back, and the result is the step-by-step one."""
    for n, radius, seeds in ((3000, 0.8, 12), (6000, 0.6, 3), (30000, 0.4, 1)):
        for s in range(seeds):
            p4 = E.single_event(n, 2 + s % 5, 1000 * n + s, **({} if n == 3000 else {"soft_mean": 0.6, "soft_eta": 4.0}))
            _check_event(ctx, p4, -1, radius, f"n {n} R {radius} seed {s}")


@pytest.mark.parametrize("algo,radius", [(-1, 1.05), (-1, 1.06), (1, 1.8), (0, 2.0), (0, 2.01)])
def test_large_radii_above_4096(ctx, algo, radius):
    """Few tiles around in azimuth (six at R = 2), and both sides of the rule's
    largest radii for events above 4096 particles."""
    _check_event(ctx, E.single_event(4200, 4, 11, soft_mean=0.6, soft_eta=4.0), algo, radius, f"algo {algo} R {radius}")
