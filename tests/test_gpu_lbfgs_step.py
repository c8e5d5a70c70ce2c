"""The L-BFGS direction kernel (lbfgs_step) through btam_relax: the iterates
against the same iteration in numpy, driven by the device's evaluations.

Sizes on both sides of the one-block line (4 n = 4096), histories shorter and
longer than the number of iterations, sites held by x_min, periodic images.
The two run the same operations; their sums differ in order, a relative
2^-52 sqrt(4 n) at most per reduction, and a step carries a difference on with
the ratio of the Hessian's extreme curvatures (some 1e3 here): over the five
iterations compared 1e-9 of the largest component bounds it."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu


def numpy_lbfgs(S, s, iters, m, x_min=0.01, lo=np.log(0.001), hi=np.log(0.4)):
    """btam_relax's mode 0 with a fixed number of iterations; (q, sigma, F, evals)."""
    x, beta = s["x"], s["beta"]
    act, rel = x >= 5e-4, (x >= 5e-4) & (x >= x_min)
    sc = np.sqrt(np.maximum(x, 1e-3))[:, None]
    evals = 0

    def gather(q, sigma):
        nonlocal evals
        evals += 1
        o = S.evaluate_state(btam.FP64, q=q, sigma=sigma)
        ls = np.log(sigma)
        gs = beta * sigma * o["Rs"]
        pin = ((ls >= hi - 1e-12) & (gs < 0)) | ((ls <= lo + 1e-12) & (gs > 0))
        z = sc * np.column_stack([q, ls])
        g = np.column_stack([beta[:, None] * o["Rq"], np.where(pin, 0.0, gs)]) / sc
        g = np.where(rel[:, None], g, 0.0)
        F = np.where(act, beta * o["V0"] - np.where(rel, 3.0 * ls, 0.0), 0.0).sum()
        r2 = np.where(rel, (o["Rq"] ** 2).sum(1) + np.where(pin, 0.0, o["Rs"] ** 2), 0.0).sum()
        return z, g, F, r2

    q, sigma = s["q"].copy(), s["sigma"].copy()
    z, g, F, r2 = gather(q, sigma)
    hist = []
    for _ in range(iters):
        d, al = g.copy(), []
        for ss, yy in reversed(hist):
            al.append((ss * d).sum() / (ss * yy).sum())
            d = d - al[-1] * yy
        if hist:
            ss, yy = hist[-1]
            d = d * ((ss * yy).sum() / (yy * yy).sum())
        for (ss, yy), a in zip(hist, reversed(al)):
            d = d + (a - (yy * d).sum() / (ss * yy).sum()) * ss
        p = -d
        gp = (g * p).sum()
        assert gp < 0  # the systems here give descent directions throughout
        step = 1.0
        if not hist:
            pmax = np.abs(p / sc).max()
            step = 0.05 / pmax if pmax > 0.05 else 1.0
        z0, g0, F0, r20 = z, g, F, r2
        for _ in range(30):
            w = (z0 + step * p) / sc
            q = np.where(rel[:, None], w[:, :3], q)
            sigma = np.where(rel, np.exp(np.clip(w[:, 3], lo, hi)), sigma)
            z, g, F, r2 = gather(q, sigma)
            if F <= F0 + 1e-4 * step * gp or (abs(F - F0) <= 1e-13 * abs(F0) and r2 < r20):
                break
            step *= 0.5
        hist.append((z - z0, g - g0))
        hist = hist[-m:]
    return q, sigma, F, evals


def periodic_cell():
    n = np.array([5, 5, 5])
    s = lattice.supercell(*n, h_fraction=0.4, x_range=(0.0, 0.5), sigma_range=(0.09, 0.12),
                          jitter=0.01, seed=12)
    # the cell's faces between the lattice planes: no iterate leaves the cell
    s["origin"] = -0.06 * (s["cell"] / n[:, None]).sum(axis=0)
    f = (s["q"] - s["origin"]) @ np.linalg.inv(s["cell"])
    s["q"] = np.ascontiguousarray((f - np.floor(f)) @ s["cell"] + s["origin"])
    return s


def open_sphere():
    return lattice.cluster("sphere", 17.5, x_fn=lambda g, r, n: g.uniform(0.0, 0.5, n),
                           sigma_range=(0.09, 0.12), h_fraction=0.4, seed=12)


@pytest.mark.parametrize("m", [2, 8])
@pytest.mark.parametrize("make", [periodic_cell, open_sphere], ids=["one_block", "cluster"])
def test_relaxation_iterates(gpu_tables, make, m):
    s = make()
    assert (4 * len(s["x"]) <= 4096) == (make is periodic_cell)
    assert np.any((s["species"] == 1) & (s["x"] < 0.01))  # held sites
    iters = 5
    D = btam.System(gpu_tables, s)
    D.build_neighbors()
    want_q, want_s, want_F, evals = numpy_lbfgs(D, s, iters, m)
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    info = S.relax(mode=btam.RELAX_FP64, tol=1e-12, max_iter=iters, m=m)
    q, sigma, _ = S.get_state()
    assert info["iterations"] == iters and info["evaluations"] == evals
    dq, ds = np.abs(q - want_q).max(), np.abs(sigma - want_s).max()
    print(make.__name__, m, evals, dq, ds, info["objective"] - want_F)
    assert dq <= 1e-9 * np.abs(want_q).max() and ds <= 1e-9
    assert abs(info["objective"] - want_F) <= 1e-10 * abs(want_F)
    # the totals left behind are those of the final state, images included
    assert np.array_equal(S.results(want=("totals",))["totals"], S.evaluate()["totals"])


@pytest.mark.parametrize("relax", [dict(mode=btam.RELAX_FP64), dict(mode=btam.RELAX_MIXED)],
                         ids=["fp64", "mixed"])
def test_totals_of_a_failed_relaxation(gpu_tables, relax):
    """An evaluation that is not finite (two occupied sites at one position) ends
    the relaxation with its error and leaves that evaluation's results, the
    totals among them."""
    s = open_sphere()
    h = np.flatnonzero((s["species"] == 1) & (s["x"] > 0.1))
    s["q"][h[1]] = s["q"][h[0]]
    prec = btam.FP64 if relax["mode"] == btam.RELAX_FP64 else btam.FP32C
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
    with pytest.raises(btam.BtamError) as want:
        R.evaluate(prec)
    with pytest.raises(btam.BtamError) as got:
        S.relax(tol=1e-8, max_iter=3, **relax)
    assert got.value.code == want.value.code == 6  # BTAM_ERR_NONFINITE
    keys = ("rho", "V0", "S0", "Rq", "Rs", "Rx", "totals")
    a, b = S.results(want=keys), R.results(want=keys)
    for k in keys:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


def test_backtracked_trials(gpu_tables):
    """A start far from a minimum, where the first trial of some iterations is
    refused and halved: same evaluations, same iterates (the tolerance above; the
    20 iterations carry a difference no further than that)."""
    s = lattice.cluster("sphere", 8.0, x_fn=lambda g, r, n: g.uniform(0.0, 0.5, n),
                        sigma_range=(0.03, 0.38), h_fraction=0.4, seed=2)
    s["q"] = s["q"] + np.random.default_rng(2).normal(0.0, 0.25, s["q"].shape)
    iters = 20
    D, S = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (D, S):
        T.build_neighbors()
    want_q, want_s, want_F, evals = numpy_lbfgs(D, s, iters, 5)
    assert evals > iters + 1
    info = S.relax(mode=btam.RELAX_FP64, tol=1e-12, max_iter=iters, m=5)
    q, sigma, _ = S.get_state()
    assert info["iterations"] == iters and info["evaluations"] == evals
    assert np.abs(q - want_q).max() <= 1e-9 * np.abs(want_q).max()
    assert np.abs(sigma - want_s).max() <= 1e-9
    assert abs(info["objective"] - want_F) <= 1e-10 * abs(want_F)
