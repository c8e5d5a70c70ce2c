"""Pass 1 of small systems, a warp per part of a site, against the one-piece
kernel.  The split runs where its blocks fit the device at once; a persistent
grid (8 of the variant) never splits.  Sums, trees and rounding are the same:
the results are equal bit for bit.  Sizes: a few sites, around one and several
blocks an SM, beyond the rule; empty sites; lists of one entry to full ones."""
import numpy as np
import pytest

import btam
from btam import lattice

pytestmark = pytest.mark.gpu


def emptied(s):
    x = s["x"].copy()
    h = np.flatnonzero(s["species"] == 1)[::4]
    x[h] = np.where(np.arange(len(h)) % 2 == 0, 1e-4, 0.0)
    return dict(s, x=x)


def half(s, n):
    keep = np.arange(len(s["x"])) < n
    return {k: v[keep] if np.ndim(v) and len(v) == len(keep) else v for k, v in s.items()}


SYSTEMS = {
    "atoms_57": lambda: lattice.cluster("sphere", 6.5, h_fraction=0.0, seed=61),
    "line_12": lambda: half(lattice.cluster("sphere", 9.0, h_fraction=0.0, seed=62), 12),
    "sphere_212": lambda: emptied(lattice.cluster("sphere", 9.0, h_fraction=0.3, seed=63)),
    "sphere_495": lambda: emptied(lattice.cluster("sphere", 11.0, h_fraction=0.5, seed=64)),
    "cell_1296": lambda: lattice.supercell(6, 6, 6, h_fraction=1.0, x_range=(0.1, 0.9),
                                           sigma_range=(0.08, 0.15), jitter=0.02, seed=65),
}


@pytest.mark.parametrize("prec", [btam.FP64, btam.FP32C])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_split_equals_one_piece(gpu_tables, name, prec):
    S = btam.System(gpu_tables, SYSTEMS[name]())
    S.build_neighbors()
    out = []
    for v1 in (16, 16 | 8):
        S.set_variants(prec, v1, 16)
        out.append(S.evaluate(prec))
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
