"""btam_mf_eval_async recorded into a CUDA graph, replayed after evaluations in
the other arithmetic form, which need a larger pair buffer.

A captured evaluation of a system that is neither tuned nor pinned is that of
the directed kernels (0, 0); one of pinned variants that of those variants, bit
for bit (a variant is reproducible).  Another system built in between, whose
memory may be what the first buffer occupied, is not disturbed."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu
KEYS = ("rho", "V0", "S0", "Rq", "Rs", "Rx", "totals")


def cell(seed, nx=5):
    return lattice.supercell(nx, 5, 5, h_fraction=0.4, x_range=(0.05, 0.6),
                             sigma_range=(0.08, 0.15), jitter=0.02, seed=seed)


def captured(torch, S, prec):
    ext = torch.cuda.ExternalStream(S.stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(ext):
        g.capture_begin(capture_error_mode="relaxed")
        status = btam.lib().btam_mf_eval_async(S.handle, prec)
        g.capture_end()
    assert status == 0
    return ext, g


@pytest.mark.parametrize("pinned", [None, (16 | 2, 16 | 1), (0, 16), (2, 1)],
                         ids=["default", "undirected", "mixed", "directed"])
def test_replay_after_the_other_form(gpu_tables, pinned):
    torch = pytest.importorskip("torch")
    s = cell(1)
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
    if pinned:
        S.set_variants(btam.FP32C, *pinned)
    R.set_variants(btam.FP32C, *(pinned or (0, 0)))
    S.evaluate(btam.FP32C)
    ext, g = captured(torch, S, btam.FP32C)
    first = S.evaluate(btam.FP64)  # takes a larger buffer
    S.set_variants(btam.FP64, 16, 16)
    S.evaluate(btam.FP64)
    S.autotune(btam.FP64)
    others = []
    for k in range(4):
        others.append(btam.System(gpu_tables, cell(2 + k, 5 + k % 2)))
        others[-1].build_neighbors()
    before = [T.evaluate(btam.FP64) for T in others]
    for f in (1.0, 1.03):
        S.set_state(sigma=s["sigma"] * f)
        R.set_state(sigma=s["sigma"] * f)
        want = R.evaluate(btam.FP32C)
        with torch.cuda.stream(ext):
            g.replay()
        got = S.results(want=KEYS)
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), (pinned, k)
        for T, b in zip(others, before):
            now = T.evaluate(btam.FP64)
            assert all(np.array_equal(now[k], b[k]) for k in KEYS)
    S.set_state(sigma=s["sigma"])
    S.set_variants(btam.FP64, 16, 16 | 0)
    again = S.evaluate(btam.FP64)  # 391 sites: the shapes the defaults took
    assert all(np.array_equal(again[k], first[k]) for k in KEYS)
    del g
