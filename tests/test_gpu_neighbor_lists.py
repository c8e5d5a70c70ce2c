"""Neighbour lists against all pairs: list lengths on both sides of every sort
size (64, 128, 256), empty cells, one row of cells, a filled box.  The distance
rule is the kernel's own, in the same order of operations: the lists are equal."""
import numpy as np
import pytest

import btam

pytestmark = pytest.mark.gpu
RC = 6.2934034034


def random_system(n, box, seed, spread=0.0):
    g = np.random.default_rng(seed)
    q = g.random((n, 3)) * np.asarray(box, float)
    if spread:  # a dense knot in one corner
        q[: n // 3] *= spread
    return dict(q=q, sigma=np.full(n, 0.1), x=np.ones(n), species=np.full(n, 12, np.int32),
                beta=np.full(n, 38.7), gamma=np.zeros(n), origin=np.zeros(3),
                cell=np.diag(np.asarray(box, float)), periodic=np.zeros(3, np.int32))


CASES = {
    "short": (60, (12.0, 12.0, 12.0), 0.0),
    "around_64": (400, (18.0, 18.0, 18.0), 0.0),
    "around_128": (1500, (22.0, 22.0, 22.0), 0.0),
    "up_to_the_cap": (1700, (19.5, 20.0, 20.0), 0.0),
    "one_row": (120, (90.0, 5.0, 5.0), 0.0),
    "knot": (500, (40.0, 40.0, 40.0), 0.35),
}


@pytest.mark.parametrize("name", list(CASES))
def test_lists_equal_all_pairs(gpu_tables, name):
    n, box, spread = CASES[name]
    s = random_system(n, box, 51, spread)
    d = s["q"][:, None, :] - s["q"][None, :, :]
    r = np.sqrt((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2])
    near = (r <= RC) & ~np.eye(n, dtype=bool)
    keep = near.any(1) if not near.any(1).all() else None
    if keep is not None:  # a site without neighbours is an error: leave those out
        s = {k: (v[keep] if np.ndim(v) and len(v) == n else v) for k, v in s.items()}
        near = near[np.ix_(keep, keep)]
    assert near.sum(1).max() <= 250
    S = btam.System(gpu_tables, s)
    S.build_neighbors()
    offs, idx = S.neighbors()
    assert np.array_equal(np.diff(offs), near.sum(1))
    assert np.array_equal(idx, np.nonzero(near)[1])
