"""Results and states on their way to the caller: one block through a pinned
slot (small systems), slots of 32,768 values in turn (larger ones), plain copies
for pinned arrays.  Every route hands over the same bits, whatever subset is
asked for, from several threads, and a rejected state leaves the old one."""
import threading

import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu
KEYS = ("rho", "V0", "S0", "Rq", "Rs", "Rx", "totals")


def system(tables, nx, ny, nz):
    s = lattice.supercell(nx, ny, nz, h_fraction=1.0, x_range=(0.1, 0.9), jitter=0.02, seed=41)
    S = btam.System(tables, s)
    S.build_neighbors()
    return S, s


def pinned_like(torch, n, k):
    shape = (4,) if k == "totals" else (n, 3) if k == "Rq" else (n,)
    return torch.zeros(shape, dtype=torch.float64).pin_memory()


# 8 n result values below one slot, just above it, and several slots an array
@pytest.mark.parametrize("dims", [(6, 6, 6), (9, 8, 8), (14, 13, 13)])
def test_every_route_hands_over_the_same_bits(gpu_tables, dims):
    torch = pytest.importorskip("torch")
    S, s = system(gpu_tables, *dims)
    n = S.n
    q, sigma = np.ascontiguousarray(s["q"]), np.asarray(s["sigma"]) * 1.01
    out = S.evaluate_state(btam.FP64, q=q, sigma=sigma, x=s["x"])
    later = S.results(want=KEYS)
    keep = {k: pinned_like(torch, n, k) for k in KEYS}
    mixed = {k: keep[k].numpy() if i % 2 else np.full(tuple(keep[k].shape), np.nan)
             for i, k in enumerate(KEYS)}
    L, d = btam.lib(), btam._d
    assert L.btam_mf_eval_state(S.handle, btam.FP64, None, None, d(s["x"]),
                                *[d(mixed[k]) for k in KEYS]) == 0
    for k in KEYS:
        assert np.array_equal(out[k], later[k]), k
        assert np.array_equal(out[k], mixed[k]), k
        assert np.array_equal(out[k], S.results(want=(k,))[k]), k
    got = S.get_state()
    for a, b in zip(got, (q, sigma, s["x"])):
        assert np.array_equal(a, b)
    bad = sigma.copy()
    bad[-1] = np.nan
    with pytest.raises(btam.BtamError):
        S.evaluate_state(btam.FP64, sigma=bad)
    assert np.array_equal(S.get_state()[1], sigma)


def test_threads_have_their_own_slots(gpu_tables):
    pairs = [system(gpu_tables, *d) for d in ((6, 6, 6), (9, 8, 8), (7, 6, 6), (10, 9, 8))]
    ref = [S.evaluate(btam.FP64) for S, _ in pairs]
    bad = []

    def work(k):
        S, s = pairs[k]
        for _ in range(8):
            o = S.evaluate_state(btam.FP64, q=s["q"], sigma=s["sigma"], x=s["x"])
            if not all(np.array_equal(o[c], ref[k][c]) for c in KEYS):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(pairs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_systems_of_one_thread_share_the_slots(gpu_tables):
    pairs = [system(gpu_tables, *d) for d in ((6, 6, 6), (7, 6, 6), (8, 6, 6))]
    for r in range(6):
        for k, (S, s) in enumerate(pairs):  # six inputs in flight, four slots
            S.set_state(sigma=s["sigma"] * (1.0 + 0.01 * (r + k)))
        for k, (S, s) in enumerate(pairs):
            assert np.array_equal(S.get_state()[1], s["sigma"] * (1.0 + 0.01 * (r + k)))


def test_threads_that_end_hand_their_slots_on(gpu_tables):
    """Jobs on threads of their own, eight at a time, each with more copies than a
    thread waits for slots of its own: the bits of one thread's."""
    dicts = [lattice.sphere(9.0 + k % 7, h_fraction=0.3, seed=k) for k in range(48)]
    bad = []

    def job(k, ref):
        S = btam.System(gpu_tables, dicts[k])
        S.build_neighbors()
        for r in range(1 + 15 * (k % 3)):
            sigma = np.asarray(dicts[k]["sigma"]) * (1.0 + 0.01 * r)
            o = S.evaluate_state(btam.FP64, sigma=sigma)
            if not np.array_equal(S.get_state()[1], sigma):
                bad.append(k)
            if ref is not None and r == 0:
                bad.extend(k for c in KEYS if not np.array_equal(o[c], ref[c]))
            if r == 0:
                first = o
        return first

    ref = [job(k, None) for k in range(len(dicts))]
    for a in range(0, len(dicts), 8):
        ts = [threading.Thread(target=job, args=(k, ref[k])) for k in range(a, a + 8)]
        for x in ts:
            x.start()
        for x in ts:
            x.join()
    assert not bad
