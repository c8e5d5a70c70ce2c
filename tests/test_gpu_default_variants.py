"""The launch variants a system or batch takes when it is neither tuned nor
pinned (default_variants): at sizes on both sides of the rule's lines, with
empty sites, open and periodic, and in a batch.

The defaults are the undirected kernels; against the directed ones (0, 0) they
agree to rounding (FP64 1e-12 relative in the energies and 1e-11 in the
residuals, FP32C 1e-6 and 1e-5, the tolerances of the launch-variant test),
and against the same shapes pinned bit for bit."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu

TOL = {btam.FP64: 1e-12, btam.FP32C: 1e-6}


def default_shapes(prec, n):
    """The rule of default_variants, restated."""
    if n < 1500:
        return 16, 16 | (0 if prec == btam.FP64 else 6)
    if prec == btam.FP64:
        return 16 | 5 | (0 if n < 20000 else 8), 16 | 6 | 8
    return 16 | (5 if n < 6000 else 2 | 8), 16 | 6 | 8


def emptied(s, every=7):
    x = s["x"].copy()
    h = np.flatnonzero(s["species"] == 1)[::every]
    x[h] = np.where(np.arange(len(h)) % 2 == 0, 1e-4, 0.0)
    return dict(s, x=x)


def cell(nx, ny, nz, h, seed):
    return emptied(lattice.supercell(nx, ny, nz, h_fraction=h, x_range=(0.0, 0.6),
                                     sigma_range=(0.08, 0.15), jitter=0.02, seed=seed))


SYSTEMS = {
    "small_cell": lambda: cell(5, 5, 5, 0.3, 1),
    "mg_only_sphere": lambda: lattice.sphere(9.0, h_fraction=0.0, seed=2),
    "cell_above_first_line": lambda: cell(7, 7, 6, 0.9, 3),
    "wire_above_second_line": lambda: lattice.wire(17.0, 8, seed=4),
}


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_defaults_against_directed_and_pinned(gpu_tables, name, prec):
    s = SYSTEMS[name]()
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    got = S.evaluate(prec)
    x_only = S.evaluate_x(prec)  # the defaults evaluate in full
    P = btam.System(gpu_tables, s)
    P.build_neighbors()
    P.set_variants(prec, *default_shapes(prec, S.n))
    pinned = P.evaluate(prec)
    P.set_variants(prec, 0, 0)
    directed = P.evaluate(prec)
    for k, v in got.items():
        assert np.array_equal(v, pinned[k]), (name, k)
        assert np.array_equal(v, x_only[k]) if k in x_only else True, (name, k)
    tol = TOL[prec]
    for k in ("rho", "V0", "S0"):
        d = np.abs(got[k] - directed[k]).max()
        assert d <= tol * max(1.0, np.abs(directed[k]).max()), (name, k, d)
    for k in ("Rq", "Rs", "Rx"):
        d = np.abs(got[k] - directed[k]).max()
        assert d <= 10 * tol * max(1.0, np.abs(directed[k]).max()), (name, k, d)


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
def test_defaults_follow_a_rebuild_and_both_forms(gpu_tables, prec):
    """A longer list after a rebuild, and one form after the other: the pair
    buffer follows."""
    s = cell(5, 5, 5, 0.3, 5)
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    other = btam.FP64 if prec == btam.FP32C else btam.FP32C
    S.evaluate(prec)
    S.evaluate(other)
    # sites pulled together lengthen the lists
    q = s["q"].copy()
    q[::3] = 0.98 * q[::3] + 0.02 * q.mean(axis=0)
    S.set_state(q=q)
    S.build_neighbors(all_sites=True)
    got = S.evaluate(prec)
    F = btam.System(gpu_tables, dict(s, q=q))
    F.build_neighbors()
    want = F.evaluate(prec)
    for k, v in got.items():
        assert np.array_equal(v, want[k]), k


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
def test_batch_defaults(gpu_tables, prec):
    systems = []
    for d in (cell(5, 5, 5, 0.3, 6), lattice.sphere(10.0, h_fraction=0.3, seed=7),
              lattice.wire(12.0, 5, seed=8)):
        systems.append(btam.System(gpu_tables, d))
        systems[-1].build_neighbors()
    B = btam.Batch(systems)
    tot = B.evaluate(prec)
    n = B.info()["n_real"]
    v1, v2 = default_shapes(prec, n)
    for k, S in enumerate(systems):
        S.set_variants(prec, v1, v2)
        want = S.evaluate(prec)
        got = B.results(k)
        for key in want:
            assert np.array_equal(got[key], want[key]), (k, key)
        assert np.array_equal(tot[k], want["totals"])
