"""The stretch relaxation's residual (pt_stress_kernel) against the point forms'
per-site stress of the stretched system.

Forms: periodic and open; empty sites; lists of a few entries, up to 64, up to 128
and beyond what a warp holds (160); fewer sites than one block and more than one round of the
grid.  No iteration is taken, so the reported norm is that of the residual at
F0, and the system is left stretched by F0, where pt_eval gives the per-site
stress.  Both sum the same FP64 terms in another order, and form r as
F (q_j - q_u) or F q_j - F q_u (an ulp of |q| <= 100 against |r| >= 2, times a
derivative of O(10)): they agree to 1e-11 of the sum of |W_u(a, a)|."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu


def emptied(s):
    x = s["x"].copy()
    h = np.flatnonzero(s["species"] == 1)[::5]
    x[h] = np.where(np.arange(len(h)) % 2 == 0, 1e-4, 0.0)
    return dict(s, x=x)


SYSTEMS = {
    "cell": lambda: emptied(lattice.supercell(5, 5, 5, h_fraction=0.6, x_range=(0.0, 0.6),
                                              jitter=0.02, seed=31)),
    "full_cell": lambda: lattice.supercell(14, 10, 8, h_fraction=1.0, x_range=(0.2, 0.9),
                                           jitter=0.02, seed=32),
    "dense_cell": lambda: lattice.supercell(9, 8, 7, h_fraction=1.0, x_range=(0.2, 0.9), a=2.75,
                                            jitter=0.01, seed=35),
    "sphere": lambda: lattice.cluster("sphere", 5.0, h_fraction=0.5, seed=33),
    "few": lambda: lattice.cluster("sphere", 3.5, h_fraction=0.0, seed=34),
}


@pytest.mark.parametrize("F0", [(1.0, 1.0, 1.0), (0.985, 1.01, 1.02)])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_residual_equals_the_point_forms_stress(gpu_tables, name, F0):
    S = btam.System(gpu_tables, SYSTEMS[name]())
    S.build_neighbors()
    _, info = S.relax_stretch(max_iter=0, F0=F0)
    assert info["evaluations"] == 1
    W = S.pt_eval()["W"]
    d = np.stack([W[:, a, a] for a in range(3)], 1) / (np.array(F0) * info["volume"])
    assert abs(info["norm"] - np.linalg.norm(d.sum(0))) <= 1e-11 * np.abs(d).sum()


@pytest.mark.parametrize("x", [0.0, 1e-4])
@pytest.mark.parametrize("name", ["cell", "full_cell", "sphere"])
def test_empty_sites_at_occupied_ones(gpu_tables, name, x):
    """An empty site at exactly the position of an occupied one weighs nothing in
    the residual, as in the point forms: same tolerance, nothing not finite."""
    s = SYSTEMS[name]()
    at = np.flatnonzero(s["x"] > 0.1)[::7]
    n = len(at)
    s = dict(s, q=np.vstack([s["q"], s["q"][at]]), sigma=np.append(s["sigma"], s["sigma"][at]),
             x=np.append(s["x"], np.full(n, x)),
             species=np.append(s["species"], np.ones(n, s["species"].dtype)),
             beta=np.append(s["beta"], s["beta"][at]), gamma=np.append(s["gamma"], np.zeros(n)))
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    F0 = (0.985, 1.01, 1.02)
    _, info = S.relax_stretch(max_iter=0, F0=F0)
    W = S.pt_eval()["W"]
    d = np.stack([W[:, a, a] for a in range(3)], 1) / (np.array(F0) * info["volume"])
    assert abs(info["norm"] - np.linalg.norm(d.sum(0))) <= 1e-11 * np.abs(d).sum()
