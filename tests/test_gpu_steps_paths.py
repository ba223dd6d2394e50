"""The step-by-step kernels where the rounds kernel takes most events: every shape and
build of the shared-memory kernel, and the tiled kernel, by calls that reach them,
against the CPU oracle bit for bit.

Shapes apply in calls of more than two events per SM, to events that the rounds
refuse (wide radii); a program in a process of its own counts them with the
phase-counter build.  The tiled kernel: wide radii, and the allocation-free entry
point, which has no workspace for the rounds.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SHAPES = {0: [(64, 4), (128, 2)], 1: [(64, 8), (128, 4), (256, 2)], 2: [(128, 8), (256, 4)],
          3: [(256, 8), (512, 4)], 4: [(512, 8), (256, 16)]}
CAPPED = [(64, 4), (64, 8), (128, 8), (256, 8)]  # shapes with a build for more CTAs per SM

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def phase_lib():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from fastjet_gpu_gb300 import build as B
    return B.build(phase_clocks=True)


@pytest.mark.parametrize("b", [0, 1, 2, 3, 4])
def test_every_shape_runs_and_is_bit_exact(phase_lib, b):
    env = dict(os.environ, FJG_LIB=phase_lib, PYTHONPATH=ROOT + os.pathsep + HERE)
    res = subprocess.run([sys.executable, os.path.abspath(__file__), str(b)], env=env, cwd=ROOT, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    for row in json.loads(res.stdout.splitlines()[-1]):
        name = "shape_%dx%d" % tuple(row["shape"])
        assert row["counts"][name] >= row["in_bucket"], row
        assert row["counts"]["r_events"] == 0 and row["counts"]["events"] == row["events"], row
        if row["ctas"] == 64 and tuple(row["shape"]) in CAPPED:
            assert row["counts"]["shape_capped"] >= row["in_bucket"], row
        if row["ctas"] == 1:
            assert row["counts"]["shape_capped"] == 0, row


def _run_noalloc(batch, algo, radius):
    import torch

    import fastjet_gpu_gb300 as F
    from test_zz_no_alloc import _run_noalloc as run
    return run(F, torch, batch, algo, radius)


def _same_as_oracle(batch, algo, radius, got):
    import oracle
    hist, jets, lab, _, nj, _ = oracle.cluster_batch(batch.particles, batch.offsets, algo, radius, threads=4,
                                                     portable=True)
    assert np.array_equal(got["n_jets"], nj)
    for k in ("a", "b", "d"):
        assert np.array_equal(got["history"][k], hist[k]), k
    for e in range(batch.n_events):
        o = batch.offsets[e]
        assert np.array_equal(got["jets"][o:o + nj[e]], jets[o:o + nj[e]]), e
        assert np.array_equal(got["jet_label"][o:o + nj[e]], lab[o:o + nj[e]]), e


# the tiled kernel's lists and summaries: sparse and dense, many tiles (R = 0.1: the cap), few
@pytest.mark.parametrize("algo,radius", [(-1, 0.4), (1, 0.6), (0, 0.8), (-1, 0.1), (1, 1.5)])
def test_tiled_kernel_without_a_workspace_for_the_rounds(phase_lib, algo, radius):
    from fastjet_gpu_gb300 import events as E
    sizes = (4097, 20000, 40000) if algo == -1 else (4097, 12000)
    evs = [E.portable_event(n, 4, seed=n + 5) for n in sizes]
    batch = E._batch_from(evs)
    assert batch.offsets[-1] <= 131072
    _same_as_oracle(batch, algo, radius, _run_noalloc(batch, algo, radius))


def test_tile_sides_of_the_tiled_kernel(phase_lib):
    """Radii that the rounds refuse above 4096 particles: each tile side gives the oracle's result."""
    import fastjet_gpu_gb300 as F
    from fastjet_gpu_gb300 import events as E
    ctx = F.Context(0)
    batch = E._batch_from([E.portable_event(n, 4, seed=n) for n in (4500, 9000)])
    for algo, radius in ((-1, 1.2), (1, 2.2)):
        for factor in (1.0, 1.5, 3.7):
            ctx.tuning = dict(ctx.tuning, tile_factor=factor)
            got = ctx.cluster_batch(batch.particles, batch.offsets, algo, radius, history=True)
            _same_as_oracle(batch, algo, radius, got)
    ctx.close()


def _main(b):
    import fastjet_gpu_gb300 as F
    from fastjet_gpu_gb300 import events as E
    ctx = F.Context(0)
    cap = 256 << b
    lo = 120 if b == 0 else cap // 2 + 1
    rng = np.random.default_rng(100 + b)
    sizes = [int(n) for n in rng.integers(lo, cap + 1, 8)] + [lo, cap] + [3 + i % 9 for i in range(310)]
    batch = E._batch_from([E.single_event(n, 3, seed=i) for i, n in enumerate(sizes)])
    rows = []
    for algo, radius in ((-1, 1.2), (1, 2.5), (0, 2.5)):
        for shape in SHAPES[b]:
            for ctas in (0, 1, 64):  # 64: as many as any build fits
                t = {k: (list(v) if isinstance(v, list) else v) for k, v in ctx.tuning.items()}
                t["threads"][b], t["slots_per_thread"][b] = shape
                t["ctas_per_sm"][b] = ctas
                ctx.tuning = t
                ctx.phase_clocks(reset=True)
                got = ctx.cluster_batch(batch.particles, batch.offsets, algo, radius, history=True)
                counts = ctx.phase_clocks()
                if shape == SHAPES[b][0] and ctas == 0:
                    _same_as_oracle(batch, algo, radius, got)
                    first = got
                for k in ("n_jets", "history"):
                    assert np.array_equal(got[k], first[k]), (algo, shape, ctas, k)
                for e in range(batch.n_events):
                    s = slice(batch.offsets[e], batch.offsets[e] + got["n_jets"][e])
                    assert np.array_equal(got["jets"][s], first["jets"][s]), (algo, shape, ctas, e)
                rows.append({"shape": shape, "ctas": ctas, "in_bucket": 10, "events": batch.n_events, "counts": counts})
    print(json.dumps(rows))


if __name__ == "__main__":
    _main(int(sys.argv[1]))
