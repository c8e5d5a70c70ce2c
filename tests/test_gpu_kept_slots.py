"""Master-equation steps on kept slot values (kept_site_kernel) against the
general x-only evaluation of the same state.

Forms: periodic and open, with empty sites, sites whose lists differ in length
down to a few entries, one beta and many, both arithmetic forms.  The kept
path forms the same terms from the same spline values; sums of a list of up to
250 terms differ in order and contraction, so the chemical potentials agree to
1e-13 (FP64) and 1e-6 (FP32C) of max(1, the largest), the tolerances of the
x-only test.  Lists that cover the images do not take the kept path: there the
two must agree to the same tolerance as well."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu

TOL = {btam.FP64: 1e-13, btam.FP32C: 1e-6}
PRM = dict(dt=1e-3, Df=0.045, dr=3.2, min_dx=1e-8, max_x=0.9)


def emptied(s, every=6):
    x = s["x"].copy()
    h = np.flatnonzero(s["species"] == 1)[::every]
    x[h] = np.where(np.arange(len(h)) % 2 == 0, 1e-4, 0.0)
    return dict(s, x=x)


def many_betas(s):
    g = np.random.default_rng(3)
    n = len(s["x"])
    return dict(s, beta=s["beta"] * g.uniform(0.8, 1.2, n), gamma=g.uniform(-0.5, 0.5, n))


def cell():
    return emptied(lattice.supercell(5, 5, 5, h_fraction=0.6, x_range=(0.0, 0.6),
                                     sigma_range=(0.08, 0.15), jitter=0.02, seed=21))


SYSTEMS = {
    "cell": cell,
    "cell_many_betas": lambda: many_betas(cell()),
    "small_sphere": lambda: emptied(lattice.cluster(
        "sphere", 5.0, x_fn=lambda g, r, n: g.uniform(0.0, 0.5, n), h_fraction=0.5, seed=22)),
    "wire": lambda: lattice.wire(9.0, 5, seed=23),
}


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_kept_potentials_equal_the_general_ones(gpu_tables, name, prec):
    s = SYSTEMS[name]()
    A = btam.System(gpu_tables, s)
    A.build_neighbors()
    A.set_variants(prec, 16 | 2, 16 | 1)
    A.dmd_setup()
    B = btam.System(gpu_tables, s)
    B.build_neighbors(all_sites=True)
    B.set_variants(prec, 16 | 2, 16 | 1)
    B.dmd_setup()
    for step in range(3):
        x, _, _ = A.dmd_occupancy()
        A.set_state(x=x)
        ref = A.evaluate_x(prec)  # the general x-only evaluation of this state
        B.set_state(x=x)
        ta, tb = A.dmd_step(1, prec, **PRM), B.dmd_step(1, prec, **PRM)
        assert ta == tb
        got = A.results(want=("rho", "V0", "Rx", "Rq", "Rs"))
        assert not np.any(got["Rq"]) and not np.any(got["Rs"])
        for k in ("rho", "V0", "Rx"):
            d = np.abs(got[k] - ref[k]).max()
            print(name, prec, step, k, d)
            assert d <= TOL[prec] * max(1.0, np.abs(ref[k]).max()), (name, k, step, d)
        xa, _, mu = A.dmd_occupancy()
        h = (s["species"] == 1) & (x >= 5e-4)
        want = ref["Rx"] + np.where(x < 0.9999, s["gamma"] / s["beta"], 0.0)
        assert np.abs(mu - want)[h].max() <= TOL[prec] * max(1.0, np.abs(want[h]).max())
        xb, Xb, _ = B.dmd_occupancy()
        # a potential's last bits move at most a few quanta's worth of x
        assert np.abs(xa - xb).max() <= 10 * TOL[prec]


@pytest.mark.parametrize("control", [False, True])
@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
@pytest.mark.parametrize("pair", [(16 | 2, 0), (16, 0 | 8), (0, 16 | 1), (2, 16 | 6 | 8)])
def test_passes_pinned_to_different_forms(gpu_tables, pair, prec, control):
    """One pass undirected, the other directed: the potentials are those of the
    directed kernels at the same state, to the launch-variant test's tolerances
    (FP64 1e-11, FP32C 1e-5), whatever was evaluated before."""
    s = cell()
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
    S.set_variants(prec, *pair)
    R.set_variants(prec, 0, 0)
    S.evaluate(prec)  # the moments of another state are there
    S.set_state(sigma=s["sigma"] * 1.1)
    S.dmd_setup()
    tol = 1e-11 if prec == btam.FP64 else 1e-5
    for _ in range(2):
        x, _, _ = S.dmd_occupancy()
        R.set_state(sigma=s["sigma"] * 1.1, x=x)
        want = R.evaluate(prec)["Rx"] + np.where(x < 0.9999, s["gamma"] / s["beta"], 0.0)
        if control:  # not divided: mu is that of the state x
            S.dmd_step_ctl(1, prec, max_dx=1.0, max_sub=1, **PRM)
        else:
            S.dmd_step(1, prec, **PRM)
        _, _, mu = S.dmd_occupancy()
        h = (s["species"] == 1) & (x >= 5e-4)
        assert np.abs(mu - want)[h].max() <= tol * max(1.0, np.abs(want[h]).max()), pair


@pytest.mark.parametrize("sub", [0, 1, 4])
@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_default_systems_keep_full_residuals(gpu_tables, name, prec, sub):
    """Neither tuned nor pinned: the steps leave the full evaluation of the state
    that the last (sub-)step moved from, bit for bit (the same default kernels),
    and move as the same steps one at a time.  sub 0: plain steps; else controlled
    ones of at most `sub` sub-steps."""
    s = SYSTEMS[name]()
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
        T.dmd_setup()
    for nsteps in (3, 1):
        m = 1
        if sub:
            total, st = S.dmd_step_ctl(nsteps, prec, max_dx=1e-6, max_sub=sub, **PRM)
            m = st["substeps"] // nsteps
            assert m == sub
        else:
            total = S.dmd_step(nsteps, prec, **PRM)
        part = dict(PRM, dt=PRM["dt"] / m)
        for k in range(nsteps * m - 1):
            R.dmd_step(1, prec, **part)
        E = btam.System(gpu_tables, s)
        E.build_neighbors()
        E.set_state(x=R.dmd_occupancy()[0])
        want = E.evaluate(prec)
        got = S.results(want=tuple(want))
        for k, v in want.items():
            assert np.array_equal(got[k], v), (name, k)
        assert np.any(got["Rq"]) and got["totals"][2] > 0.0
        assert R.dmd_step(1, prec, **part) == total
        assert np.array_equal(S.dmd_occupancy()[1], R.dmd_occupancy()[1])


@pytest.mark.parametrize("variants", [None, (16 | 2, 16 | 1)], ids=["default", "pinned"])
@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
def test_results_of_a_refused_step(gpu_tables, prec, variants):
    """A controlled step whose ratios are not finite ends with that error and
    leaves the results of the evaluation it rests on: in full for a system left
    to the defaults (bit for bit), its energies for pinned variants (to the
    x-only test's tolerance of rho, V0 and S0 between the two forms)."""
    s = cell()
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
        if variants:
            T.set_variants(prec, *variants)
    S.evaluate(prec)
    S.dmd_setup()
    S.set_state(sigma=s["sigma"] * 1.1)
    with pytest.raises(btam.BtamError) as e:
        S.dmd_step_ctl(2, prec, **dict(PRM, dt=1e308))
    assert e.value.code == 6  # BTAM_ERR_NONFINITE
    R.set_state(sigma=s["sigma"] * 1.1, x=S.dmd_occupancy()[0])
    want = R.evaluate(prec)
    got = S.results(want=tuple(want))
    if variants is None:
        for k, v in want.items():
            assert np.array_equal(got[k], v), k
    else:
        for c in (0, 1):
            assert abs(got["totals"][c] - want["totals"][c]) <= TOL[prec] * abs(want["totals"][c])


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
def test_results_of_a_refused_run(gpu_tables, prec):
    """The same in a run that would relax after its steps."""
    s = cell()
    S, R = btam.System(gpu_tables, s), btam.System(gpu_tables, s)
    for T in (S, R):
        T.build_neighbors()
    S.dmd_setup()
    with pytest.raises(btam.BtamError) as e:
        S.dmd_run(2, prec, relax_every=1, relax_max_iter=2, **dict(PRM, dt=1e308))
    assert e.value.code == 6
    R.set_state(x=S.dmd_occupancy()[0])
    want = R.evaluate(prec)
    got = S.results(want=tuple(want))
    for k, v in want.items():
        assert np.array_equal(got[k], v), k


def test_kept_values_are_bounded(gpu_tables):
    """Steps of a system whose kept values would exceed 4 GB leave no more than
    their small arrays in the library's pool (256 MB), and move as the general
    evaluation says (the x-only test's tolerance)."""
    torch = pytest.importorskip("torch")
    s = lattice.supercell(30, 28, 24, h_fraction=1.0, x_range=(0.1, 0.6), seed=24)
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    S.set_variants(btam.FP64, 16 | 5, 16 | 6)
    ref = S.evaluate_x(btam.FP64)["Rx"] + s["gamma"] / s["beta"]
    S.dmd_setup()
    assert S.neighbors()[1].size * 36 * 8 > (4 << 30)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    S.dmd_step(1, btam.FP64, **dict(PRM, dt=0.0))
    h = s["species"] == 1
    mu = S.dmd_occupancy()[2][h]
    assert np.abs(mu - ref[h]).max() <= TOL[btam.FP64] * max(1.0, np.abs(ref[h]).max())
    S.dmd_step(2, btam.FP64, **PRM)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 256 << 20
