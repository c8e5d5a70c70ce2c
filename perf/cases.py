"""Performance cases: the calls a user of the package makes, through its public
Python entry points, over the range of system sizes it is used on.

A case is a dict of plain values; `listed()` returns the fixed ones, `draw`
makes more of the same ranges, `prepare` builds what a program holds before
the call, `run` makes one call, `work` states what the call cannot do without
and `exact` restates the result in 64-bit torch from the table files alone.

Systems are hcp Mg with hydrogen on tetrahedral sites: the periodic cells, the
nanowire and the spheres of the repository's workloads, drawn from a seed.
FP32C results carry single precision in float64 arrays; they are handed on as
float32, as a program that stores them would keep them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bt-am_b200"))
import btam  # noqa: E402

A, C = 3.209, 3.209 * 1.624
RC = btam.R_CUTOFF
KB = 8.617332478e-5
PREC = {"fp64": btam.FP64, "fp32c": btam.FP32C}

# hexagonal 2-atom cell: Mg sites, then the tetrahedral interstitial sites
_HEX = np.array([[A, 0.0, 0.0], [-0.5 * A, 0.5 * math.sqrt(3.0) * A, 0.0], [0.0, 0.0, C]])
_MG = np.array([[0.0, 0.0, 0.0], [1.0 / 3.0, 2.0 / 3.0, 0.5]])
_TET = np.array([[0.0, 0.0, 3.0 / 8.0], [0.0, 0.0, 5.0 / 8.0],
                 [1.0 / 3.0, 2.0 / 3.0, 1.0 / 8.0], [1.0 / 3.0, 2.0 / 3.0, 7.0 / 8.0]])


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest call: one residual evaluation of a new state of a
        # 250-Mg periodic cell (a unit-test sized or teaching system, and what
        # every small served job repeats): launches and copies count
        dict(name="eval_cell_fp64", kind="eval", shape="hex", nx=5, ny=5, nz=5, h=0.2, xmax=0.1,
             prec="fp64", tuned=False),
        # the drop-in workload: 9,000 Mg and 18,000 H sites, FP64, kernel
        # shapes tuned once as a solver loop does
        dict(name="eval_cube_fp64", kind="eval", shape="hex", nx=20, ny=15, nz=15, h=1.0,
             xmax=0.3, prec="fp64", tuned=True),
        # the same in the FP32 form with compensated sums
        dict(name="eval_cube_fp32c", kind="eval", shape="hex", nx=20, ny=15, nz=15, h=1.0,
             xmax=0.3, prec="fp32c", tuned=True),
        # the largest cell of the served range (60,000 Mg), without tuning:
        # what a caller of evaluate alone gets
        dict(name="eval_large_fp64", kind="eval", shape="hex", nx=31, ny=31, nz=31, h=0.3,
             xmax=0.3, prec="fp64", tuned=False),
        # a moved nanowire: new positions, new neighbour lists, one evaluation
        # (the first evaluation of every job, and after every rebuild)
        dict(name="rebuild_wire_fp32c", kind="rebuild", shape="wire", R=20.0, length=13, h=1.0,
             xmax=0.5, prec="fp32c", tuned=False),
        # the batched form: 128 spheres of 90 to 2,800 Mg in one evaluation
        dict(name="batch_spheres_fp32c", kind="batch", n_sys=128, prec="fp32c", tuned=True),
        # master-equation steps of the nanowire of the precision workload
        dict(name="dmd_wire_fp32c", kind="dmd", shape="wire", R=30.0, length=20, h=1.0, xmax=0.5,
             prec="fp32c", tuned=True, nsteps=10, control=False),
        # step-controlled master-equation steps of a small cell in FP64
        dict(name="dmd_cell_fp64", kind="dmd", shape="hex", nx=9, ny=9, nz=9, h=0.5, xmax=0.3,
             prec="fp64", tuned=False, nsteps=10, control=True),
        # relaxation of q and sigma (L-BFGS) of a small cell: many short
        # evaluations and vector operations, launch bound
        dict(name="relax_cell_fp64", kind="relax", shape="hex", nx=6, ny=6, nz=6, h=0.2,
             xmax=0.1, prec="fp64", tuned=False, iters=15),
        # and of the drop-in system
        dict(name="relax_cube_fp64", kind="relax", shape="hex", nx=20, ny=15, nz=15, h=1.0,
             xmax=0.3, prec="fp64", tuned=True, iters=10),
        # the reference's own solver: the bulk stretch relaxation on the
        # non-mean-field stress, then the point forms of the relaxed cell
        dict(name="stretch_cube_fp64", kind="stretch", shape="hex", nx=20, ny=15, nz=15, h=1.0,
             xmax=0.3, prec="fp64", tuned=False),
        # the served form: relaxation and master-equation jobs of mixed sizes
        # submitted together, each admitted, built, run and collected
        dict(name="serve_mix", kind="serve", jobs=16, mg_lo=250, mg_hi=6000, prec="fp32c",
             tuned=False, nsteps=20, iters=8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_cell(rng, lo, hi):
    """A periodic cell of lo to hi Mg (log-uniform), at least 2 rc thick."""
    n = _log(rng, lo, hi)
    if rng.random() < 0.3:  # orthogonal cell, 4 Mg each
        dims = np.array([A, math.sqrt(3.0) * A, C])
        e = (n / 4.0 * dims.prod()) ** (1.0 / 3.0)
        k = [max(m, int(round(e / d * rng.uniform(0.8, 1.25)))) for d, m in zip(dims, (4, 3, 3))]
        return dict(shape="ortho", nx=k[0], ny=k[1], nz=k[2])
    e = (n / 2.0) ** (1.0 / 3.0)
    k = [max(5, int(round(e * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    return dict(shape="hex", nx=k[0], ny=k[1], nz=k[2])


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "eval", "rebuild", "batch", "dmd", "dmd", "relax",
                       "relax", "stretch", "serve"])
    prec = rng.choice(["fp64", "fp32c"])
    h, xmax = round(rng.uniform(0.05, 1.0), 3), round(rng.uniform(0.1, 0.5), 3)
    shape = rng.choice(["cell", "cell", "wire", "sphere"])
    if kind == "stretch":
        shape, prec = "cell", "fp64"
    if kind == "relax":
        prec = "fp64"
    hi = 20000 if kind == "eval" else 9000 if kind in ("rebuild", "dmd", "relax", "stretch") else 0
    if kind == "batch":
        return dict(kind=kind, n_sys=rng.randint(9, 120), prec=prec, tuned=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind=kind, jobs=rng.randint(5, 14), mg_lo=250, mg_hi=rng.randint(1000, 6000),
                    prec=prec, tuned=False, nsteps=rng.randint(5, 20), iters=rng.randint(4, 8))
    if shape == "cell":
        c = _draw_cell(rng, 250, hi)
    elif shape == "wire":
        c = dict(shape="wire", R=round(_log(rng, 9.0, 27.0), 2), length=rng.randint(4, 19))
    else:
        c = dict(shape="sphere", R=round(_log(rng, 8.0, 25.0), 2))
    c.update(kind=kind, h=h, xmax=xmax, prec=prec, tuned=rng.random() < 0.5)
    if kind == "dmd":
        c.update(nsteps=rng.randint(3, 12), control=rng.random() < 0.4)
    if kind == "relax":
        c.update(iters=rng.randint(4, 10))
    return c


# ---------------------------------------------------------------------------
# inputs

def _lattice(case):
    """Mg and tetrahedral positions with the cell of a case, before seeding."""
    if case["shape"] in ("hex", "ortho"):
        n = np.array([case["nx"], case["ny"], case["nz"]])
        if case["shape"] == "hex":
            vec, mg, tet = _HEX, _MG, _TET
        else:  # a x sqrt(3) a x c: the hexagonal sites twice
            vec = np.diag([A, math.sqrt(3.0) * A, C])
            inv = np.linalg.inv(vec)
            two = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.0]])
            mg, tet = (((b @ _HEX @ inv)[None] + two[:, None]).reshape(-1, 3) % 1.0
                       for b in (_MG, _TET))
        k, j, i = np.meshgrid(*(np.arange(m) for m in n[::-1]), indexing="ij")
        cells = np.stack([i, j, k], -1).reshape(-1, 3).astype(float)
        q = [(cells[:, None] + b[None]).reshape(-1, 3) @ vec for b in (mg, tet)]
        return q[0], q[1], vec * n[:, None], np.zeros(3), np.array([1, 1, 1])
    R, wire = case["R"], case["shape"] == "wire"
    m = int(math.ceil(R / A)) + 2
    nz = np.arange(case["length"]) if wire else np.arange(-int(R / C) - 2, int(R / C) + 3)
    k, j, i = np.meshgrid(nz, np.arange(-2 * m, 2 * m + 1), np.arange(-2 * m, 2 * m + 1),
                          indexing="ij")
    cells = np.stack([i, j, k], -1).reshape(-1, 3).astype(float)
    q = []
    for b in (_MG, _TET):
        p = (cells[:, None] + b[None]).reshape(-1, 3) @ _HEX
        r = np.hypot(p[:, 0], p[:, 1]) if wire else np.linalg.norm(p, axis=1)
        q.append(p[r <= R])
    every = np.concatenate(q)
    lo, hi = every.min(0) - 2.0, every.max(0) + 2.0
    if wire:
        lo[2], hi[2] = 0.0, case["length"] * C
    return q[0], q[1], np.diag(hi - lo), lo, np.array([0, 0, 1 if wire else 0])


def system(case, seed):
    """The seeded system of a case: jittered positions, widths on [0.08, 0.15],
    hydrogen on a fraction h of the tetrahedral sites with x on [0.01, xmax]."""
    g = np.random.default_rng([int(seed), 17])
    mg, tet, cell, origin, periodic = _lattice(case)
    keep = max(1, int(round(case["h"] * len(tet))))  # the same number for every seed
    tet = tet[np.sort(g.permutation(len(tet))[:keep])]
    q = np.concatenate([mg, tet])
    q = q + g.normal(0.0, 0.02, q.shape)
    n = len(q)
    if periodic.any():  # into the cell
        f = (q - origin) @ np.linalg.inv(cell)
        q = np.where(periodic, f - np.floor(f), f) @ cell + origin
    x = np.concatenate([np.ones(len(mg)), g.uniform(0.01, case["xmax"], len(tet))])
    T = float(g.uniform(300.0, 600.0))
    return dict(q=np.ascontiguousarray(q), sigma=g.uniform(0.08, 0.15, n), x=x,
                species=np.concatenate([np.full(len(mg), 12), np.full(len(tet), 1)]).astype(
                    np.int32),
                beta=np.full(n, 1.0 / (KB * T)), gamma=np.zeros(n), origin=origin, cell=cell,
                periodic=periodic.astype(np.int32))


def _batch_systems(case, seed):
    """Spheres with radii spread over the logarithm of [8, 25] A and H fractions
    up to 1/2."""
    g, size = np.random.default_rng([int(seed), 29]), np.random.default_rng(case["n_sys"])
    R = np.exp(np.linspace(math.log(8.0), math.log(25.0), case["n_sys"]))
    return [system(dict(shape="sphere", R=float(r), h=float(size.uniform(0.05, 0.5)), xmax=0.5),
                   g.integers(1 << 30)) for r in size.permutation(R)]


def _serve_jobs(case, seed):
    """(system, is relaxation) of a served mix: cells, wires and spheres."""
    g, size = np.random.default_rng([int(seed), 31]), np.random.default_rng(case["jobs"])
    jobs = []
    for k in range(case["jobs"]):
        n = float(np.exp(size.uniform(math.log(case["mg_lo"]), math.log(case["mg_hi"]))))
        e = max(5, int(round((n / 2.0) ** (1.0 / 3.0))))
        c = [dict(shape="hex", nx=e, ny=e, nz=e), dict(shape="hex", nx=e, ny=e, nz=e),
             dict(shape="wire", R=10.0 + 2.0 * (k % 5), length=4 + k % 7),
             dict(shape="sphere", R=float(min(25.0, 1.77 * n ** (1.0 / 3.0))))][k % 4]
        c.update(h=float(size.uniform(0.05, 0.5)), xmax=0.3)
        jobs.append((system(c, g.integers(1 << 30)), k % 2 == 0))
    return jobs


_TABLES = []


def tables():
    """The potential, loaded once per program."""
    if not _TABLES:
        _TABLES.append(btam.Tables())
    return _TABLES[0]


def _built(sysdict, case):
    S = btam.System(tables(), sysdict)
    S.build_neighbors()
    if case["tuned"]:
        S.autotune(PREC[case["prec"]])
    return S


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems = [_built(s, dict(case, tuned=False)) for s in _batch_systems(case, seed)]
        B = btam.Batch(systems)
        if case["tuned"]:
            B.autotune(PREC[case["prec"]])
        return dict(case=case, B=B)
    if kind == "serve":
        return dict(case=case, server=btam.Server(tables(), workers=8),
                    jobs=_serve_jobs(case, seed))
    s = system(case, seed)
    S = _built(s, case)
    if kind == "dmd":
        S.dmd_setup()
    return dict(case=case, S=S, q=s["q"], sigma=s["sigma"], x=s["x"])


# ---------------------------------------------------------------------------
# one call

def _kept(out, case):
    """FP32C results as the single precision they carry."""
    if case["prec"] == "fp64":
        return out
    return {k: v.astype(np.float32) for k, v in out.items()}


def run(state):
    case = state["case"]
    kind, prec = case["kind"], PREC[case["prec"]]
    if kind == "batch":
        return _kept(dict(totals=state["B"].evaluate(prec)), case)
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(s, btam.JOB_RELAX, precision=btam.FP64, mode=btam.RELAX_FP64, tol=1e-8,
                          max_iter=case["iters"]) if relax else
               srv.submit(s, btam.JOB_DMD, precision=prec, nsteps=case["nsteps"])
               for s, relax in state["jobs"]]
        out = []
        for job, (_, relax) in zip(ids, state["jobs"]):
            r = srv.wait(job)
            out.append(dict(q=r["q"], sigma=r["sigma"], energy=float(r["objective"])) if relax else
                       _kept(dict(x=r["x"]), case))
        return out
    S = state["S"]
    if kind == "eval":
        return _kept(S.evaluate_state(prec, q=state["q"], sigma=state["sigma"], x=state["x"]),
                     case)
    if kind == "rebuild":
        S.set_state(q=state["q"])
        S.build_neighbors()
        return _kept(S.evaluate(prec), case)
    if kind == "dmd":
        if case["control"]:
            S.dmd_step_ctl(case["nsteps"], prec, dt=1e-3)
        else:
            S.dmd_step(case["nsteps"], prec, dt=1e-3)
        x, _, mu = S.dmd_occupancy()
        return _kept(dict(x=x, mu=mu), case)
    if kind == "relax":
        S.set_state(q=state["q"], sigma=state["sigma"])
        info = S.relax(mode=btam.RELAX_FP64, tol=1e-8, max_iter=case["iters"])
        q, sigma, _ = S.get_state()
        return dict(q=q, sigma=sigma, objective=float(info["objective"]))
    F, _ = S.relax_stretch()
    out = S.pt_eval()
    S.stretch(1.0 / F)  # back to the unstrained cell, for the next call
    return dict(F=F, rho=out["rho"], V=out["V"], Fq=out["Fq"], W=out["W"])


# ---------------------------------------------------------------------------
# what a call cannot do without

def _counts(case):
    """Sites and directed neighbour pairs, from the volume (surfaces ignored)."""
    vol = abs(np.linalg.det(_HEX))
    if case["shape"] in ("hex", "ortho"):
        cells = case["nx"] * case["ny"] * case["nz"] * (2 if case["shape"] == "ortho" else 1)
    elif case["shape"] == "wire":
        cells = math.pi * case["R"] ** 2 * case["length"] * C / vol
    else:
        cells = 4.0 / 3.0 * math.pi * case["R"] ** 3 / vol
    per = 2.0 + 4.0 * case["h"]
    n = cells * per
    return n, n * per / vol * 4.0 / 3.0 * math.pi * RC ** 3


def work(case):
    """Bytes: the state read (5 doubles a site) and the results written (8), per
    evaluation, and each neighbour index once where lists are built.  Operations:
    1,500 per directed pair and evaluation (25 quadrature geometries per
    undirected pair at about 110 each), 500 for the chemical potentials alone
    (the 13 triplet geometries without derivatives, the pair rule kept), 150 for
    the point forms (one geometry each way)."""
    kind = case["kind"]
    if kind == "batch":
        r = np.exp(np.linspace(math.log(8.0), math.log(25.0), case["n_sys"]))
        c = [_counts(dict(shape="sphere", R=float(v), h=0.275)) for v in r]
        n, p = (sum(v) for v in zip(*c))
        return dict(bytes=n * 13 * 8, flops=p * 1500.0)
    if kind == "serve":
        e = np.exp(np.linspace(math.log(case["mg_lo"]), math.log(case["mg_hi"]), case["jobs"]))
        n = float(e.sum()) * 1.55
        p = n * 3.1 / abs(np.linalg.det(_HEX)) * 4.0 / 3.0 * math.pi * RC ** 3
        evals = 0.5 * case["iters"], 0.5 * case["nsteps"]
        return dict(bytes=n * 13 * 8 * sum(evals) + 4 * p,
                    flops=p * (1500.0 * evals[0] + 500.0 * evals[1]))
    n, p = _counts(case)
    state = n * 13 * 8
    if kind == "eval":
        return dict(bytes=state, flops=p * 1500.0)
    if kind == "rebuild":
        return dict(bytes=state + 4 * p, flops=p * 1510.0)
    if kind == "dmd":
        return dict(bytes=state * case["nsteps"], flops=p * 500.0 * case["nsteps"])
    if kind == "relax":
        return dict(bytes=state * case["iters"], flops=p * 1500.0 * case["iters"])
    return dict(bytes=n * 17 * 8 * 5, flops=p * 150.0 * 5)


# ---------------------------------------------------------------------------
# the results in 64 bits, from the table files alone

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


_SPLINES = {}


def _splines():
    """name -> (dx, coefficients (n, 4)): rho and F of Mg and H, phi, u, w of
    the pair kinds 0 Mg-Mg, 1 H-H, 2 Mg-H."""
    if _SPLINES:
        return _SPLINES
    base = os.path.join(os.getcwd(), "bt-am_b200", "data")
    for file, kind, names in (("adpmg.dat", 0, ("rho", "F", "phi", "u", "w")),
                              ("adph.dat", 1, ("rho", "F", "phi", "u", "w")),
                              ("adpmgh.dat", 2, ("phi", "u", "w"))):
        with open(os.path.join(base, file)) as f:
            v = f.read().split()
        at = 1 if kind == 2 else 3
        if kind != 2:
            _SPLINES["mass", kind] = float(v[0])
        for name in names:
            n, dx = int(v[at]), float(v[at + 1])
            rows = np.array(v[at + 2:at + 2 + 9 * n], np.float64).reshape(n, 9)[:, :4]
            _SPLINES[name, kind] = dx, torch.from_numpy(rows.copy()).to(_device())
            at += 2 + 9 * n
    return _SPLINES


def _eval_spline(tab, kind, r):
    """Cubic of each entry's own table at r (tables of `tab` share their knots);
    the argument is held to the last knot, the slope is the cubic's there."""
    dx = tab[0][0]
    c = torch.stack([t[1] for t in tab])
    r0 = r.detach()
    m = torch.clamp(torch.floor(r0 / dx).long(), 0, c.shape[1] - 1)
    p = torch.clamp(r0 - m.to(r0.dtype) * dx, max=dx)
    k = c[kind, m]
    v = k[..., 0] + (k[..., 1] + (k[..., 2] + k[..., 3] * p) * p) * p
    d = k[..., 1] + (2.0 * k[..., 2] + 3.0 * k[..., 3] * p) * p
    return v + d * (r - r0)


def _pairs(q, cell, origin, periodic):
    """Directed pairs (i, j, shift) within the cutoff, sites binned in cells of
    at least that edge; a cell is at least two cutoffs thick, so each site
    meets at most one image of another."""
    n, dev = len(q), q.device
    inv = torch.linalg.inv(cell)
    per = torch.as_tensor(np.asarray(periodic, np.float64), device=dev)
    ii, jj, sh = [], [], []
    step = max(1, int(4e7 // n))
    for a in range(0, n, step):
        d = q[a:a + step, None] - q[None]
        f = torch.round(d @ inv) * per
        s = f @ cell
        r2 = (d - s).square().sum(-1)
        i, j = torch.nonzero(r2 <= RC * RC, as_tuple=True)
        keep = (i + a) != j
        i, j = i[keep], j[keep]
        ii.append(i + a)
        jj.append(j)
        sh.append(s[i, j])
        del d, f, s, r2
    return torch.cat(ii), torch.cat(jj), torch.cat(sh)


def _bilinear(a, la, b, lb):
    tr = la.diagonal(dim1=-2, dim2=-1).sum(-1) * lb.diagonal(dim1=-2, dim2=-1).sum(-1)
    return 0.5 * (a * b).sum(-1) + 0.5 * (la * lb).sum((-2, -1)) - tr / 6.0


class _Model:
    """Mean-field and point energies of one system in torch float64."""

    def __init__(self, s):
        dev = _device()
        T = _splines()
        self.n = len(s["x"])
        self.q, self.sigma, self.x = (torch.from_numpy(np.array(s[k])).to(dev)
                                      for k in ("q", "sigma", "x"))
        self.beta, self.gamma = (torch.from_numpy(np.array(s[k])).to(dev)
                                 for k in ("beta", "gamma"))
        self.h = torch.from_numpy((s["species"] == 1).astype(np.int64)).to(dev)
        cell = torch.from_numpy(np.array(s["cell"], np.float64)).to(dev)
        self.i, self.j, self.shift = _pairs(self.q, cell, s["origin"], s["periodic"])
        self.cell = cell
        hi, hj = self.h[self.i], self.h[self.j]
        self.kind = torch.where(hi == hj, hi, torch.full_like(hi, 2))
        self.T = T
        self.mass = torch.tensor([T["mass", 0], T["mass", 1]], dtype=torch.float64, device=dev)
        order = torch.searchsorted(self.i, torch.arange(self.n + 1, device=dev))
        self.first = order.tolist()

    def _tab(self, name):
        return [self.T[name, k] for k in range(3)] if name in ("phi", "u", "w") else \
            [self.T[name, k] for k in range(2)]

    def energies(self, q, sigma, x, lo, hi, mean_field=True):
        """(rho, V) of sites lo..hi."""
        e = slice(self.first[lo], self.first[hi])
        i, j, kind = self.i[e], self.j[e], self.kind[e]
        m = hi - lo
        live = ((x.detach()[i] >= btam.MIN_OCCUPANCY) & (x.detach()[j] >= btam.MIN_OCCUPANCY))
        i, j, kind, shift = i[live], j[live], kind[live], self.shift[e][live]
        at = i - lo
        r0 = q[i] - q[j] - shift
        X = x[i] * x[j]
        dev = q.device

        def total(v):
            return torch.zeros((m,) + v.shape[1:], dtype=v.dtype, device=dev).index_add(0, at, v)

        def feature(r):
            d = r.norm(dim=-1)
            u = X * _eval_spline(self._tab("u"), kind, d)
            w = X * _eval_spline(self._tab("w"), kind, d)
            return u[:, None] * r, w[:, None, None] * r[:, :, None] * r[:, None, :]

        def pair(r):
            d = r.norm(dim=-1)
            return (x[j] * _eval_spline(self._tab("rho"), self.h[j], d),
                    0.5 * X * _eval_spline(self._tab("phi"), kind, d))

        eye = torch.eye(3, dtype=torch.float64, device=dev)
        f0 = feature(r0)
        G0 = [total(v) for v in f0]
        if not mean_field:
            rho, phi = (total(v) for v in pair(r0))
            ang = _bilinear(*G0, *G0)
        else:
            rho = phi = diag = ang = 0.0
            H = [torch.zeros_like(v) for v in G0]
            for k in range(3):
                for sg in (1.0, -1.0):
                    for s in (sigma[i], sigma[j]):
                        r = r0 + (sg * math.sqrt(6.0) * s)[:, None] * eye[k]
                        a, b = pair(r)
                        f = feature(r)
                        rho = rho + total(a) / 12.0
                        phi = phi + total(b) / 12.0
                        diag = diag + total(_bilinear(*f, *f)) / 12.0
                    f = feature(r0 + (sg * 3.0 * sigma[i])[:, None] * eye[k])
                    G = [total(v) for v in f]
                    ang = ang + (_bilinear(*G, *G) - total(_bilinear(*f, *f))) / 18.0
                    f = feature(r0 + (sg * 3.0 * sigma[j])[:, None] * eye[k])
                    H = [t + total(v) for t, v in zip(H, f)]
                    ang = ang - total(_bilinear(*f, *f0)) / 9.0
            ang = ang + _bilinear(*H, *G0) / 9.0 + diag
        emb = _eval_spline(self._tab("F"), self.h[lo:hi], rho)
        return rho, x[lo:hi] * emb + phi + ang

    def evaluate(self, x=None):
        """rho, V0, S0, Rq, Rs, Rx and totals, as numpy."""
        q, sigma = self.q.clone().requires_grad_(), self.sigma.clone().requires_grad_()
        x = (self.x if x is None else x).clone().requires_grad_()
        n, rho, V = self.n, [], []
        step = max(1, int(n * 1.5e5 / max(1, len(self.i))))
        for a in range(0, n, step):
            r, v = self.energies(q, sigma, x, a, min(n, a + step))
            (self.beta[a:a + step] * v).sum().backward()
            rho.append(r.detach())
            V.append(v.detach())
        rho, V, b = torch.cat(rho), torch.cat(V), self.beta
        Rq, Rs, Rx = q.grad / b[:, None], sigma.grad / b, x.grad / b
        x = x.detach()
        act, one = x >= btam.MIN_OCCUPANCY, x < 1.0
        m = 103.4993333e-6 * x * self.mass[self.h]
        log_z = 3.0 * torch.log(self.sigma * torch.sqrt(m / b) / 6.5821192815e-4)
        log_z = log_z + torch.where(one, -torch.log(torch.where(one, 1.0 - x, x)), 0.0 * x)
        S = -log_z + 0.5 + b * V - self.gamma * x * self.h
        Rs = Rs - 3.0 / (b * self.sigma)
        inner = 1.5 / x + torch.where(one, 1.0 / torch.where(one, 1.0 - x, x), 0.0 * x)
        Rx = (Rx - inner / b - torch.where(x < 0.9999, self.gamma / b, 0.0 * x)) * self.h
        out = dict(rho=rho, V0=V, S0=S, Rq=Rq * act[:, None], Rs=Rs * act, Rx=Rx * act)
        out["totals"] = torch.stack([V.sum(), S.sum(), (out["Rq"] ** 2).sum() +
                                     (out["Rs"] ** 2).sum(), (out["Rx"] ** 2).sum()])
        return {k: v.cpu().numpy() for k, v in out.items()}

    def point(self, F):
        """rho, V, Fq, W of the point forms at q = diag(F) q0, as torch."""
        n = self.n
        cols = [torch.zeros(n, 3, dtype=torch.float64, device=self.q.device),
                torch.zeros(n, 3, 3, dtype=torch.float64, device=self.q.device)]
        shift0, rho, V = self.shift, [], []
        step = max(1, int(n * 2e6 / max(1, len(self.i))))
        for a in range(0, n, step):
            b = min(n, a + step)
            e = slice(self.first[a], self.first[b])
            i, j = self.i[e], self.j[e]
            edge = ((self.q[i] - self.q[j] - shift0[e]) * F).requires_grad_()
            # each edge its own variable: site 0 of pair k at edge k, site 1 at 0
            r, v = _Edges(self, a, b, e).energies(edge)
            g, = torch.autograd.grad(v.sum(), edge)  # dV_i / d(q_i - q_j)
            cols[0].index_add_(0, i, g)
            cols[0].index_add_(0, j, -g)
            cols[1].index_add_(0, i, g[:, :, None] * edge.detach()[:, None, :])
            rho.append(r.detach())
            V.append(v.detach())
        return torch.cat(rho), torch.cat(V), cols[0], cols[1]


class _Edges:
    """The point energies of sites a..b as functions of their edge vectors."""

    def __init__(self, model, a, b, e):
        self.m, self.a, self.b, self.e = model, a, b, e

    def energies(self, edge):
        M, lo, hi, e = self.m, self.a, self.b, self.e
        i, j, kind, x = M.i[e] - lo, M.j[e], M.kind[e], M.x
        X = x[M.i[e]] * x[j]
        d = edge.norm(dim=-1)

        def total(v):
            return torch.zeros((hi - lo,) + v.shape[1:], dtype=v.dtype,
                               device=v.device).index_add(0, i, v)

        u, w = (X * _eval_spline(M._tab(k), kind, d) for k in ("u", "w"))
        G = (total(u[:, None] * edge), total(w[:, None, None] * edge[:, :, None] *
                                             edge[:, None, :]))
        rho = total(x[j] * _eval_spline(M._tab("rho"), M.h[j], d))
        phi = total(0.5 * X * _eval_spline(M._tab("phi"), kind, d))
        return rho, x[lo:hi] * _eval_spline(M._tab("F"), M.h[lo:hi], rho) + phi + \
            _bilinear(*G, *G)


def _exact_stretch(s):
    """The stretch that zeroes the mean stress (Newton on the three components)
    and the point forms there."""
    M = _Model(s)
    F = torch.ones(3, dtype=torch.float64, device=M.q.device)
    stress = lambda f: M.point(f)[3].sum(0).diagonal() / f  # noqa: E731
    for _ in range(8):
        y = stress(F)
        J = torch.stack([(stress(F + 1e-5 * e) - stress(F - 1e-5 * e)) / 2e-5
                         for e in torch.eye(3, dtype=torch.float64, device=F.device)], 1)
        F = F - torch.linalg.solve(J, y)
    rho, V, Fq, W = M.point(F)
    return dict(F=F.cpu().numpy(), rho=rho.cpu().numpy(), V=V.cpu().numpy(), Fq=Fq.cpu().numpy(),
                W=W.cpu().numpy())


def _exact_dmd(s, nsteps, control, dt=1e-3, Df=0.045, dr=3.2, min_dx=1e-8, max_x=0.9,
               max_dx=0.05, max_sub=64):
    """Occupancies and last chemical potentials of the master equation on the
    H-H graph (2.6 A): each edge moves dt Df / dr^2 beta xm (1 - xm) (mu_i -
    mu_j), held to the room its ends have."""
    M = _Model(s)
    H, n = M.h == 1, M.n
    d2 = (M.q[M.i] - M.q[M.j] - M.shift).square().sum(-1)
    edge = H[M.i] & H[M.j] & (d2 <= 2.6 ** 2)
    ei, ej = M.i[edge], M.j[edge]
    once = ei < ej
    ei, ej = ei[once], ej[once]
    hh = H[M.i] & H[M.j]
    x = M.x.clone()
    zero = torch.zeros_like(x)

    def potential():
        Rx = torch.from_numpy(M.evaluate(x)["Rx"]).to(x.device)
        low = torch.clamp(x, min=1e-12)
        mu = torch.where(x >= btam.MIN_OCCUPANCY,
                         Rx + torch.where(x < 0.9999, M.gamma / M.beta, zero),
                         -(1.5 / low + 1.0 / (1.0 - torch.where(H, low, zero))) / M.beta)
        mass = (x * H).index_add(0, M.i[hh], x[M.j[hh]])
        return torch.where(H, mu, zero), H & (mass >= 0.01)

    def moves(mu, act, step):
        on = act[ei] & act[ej]
        i, j = ei[on], ej[on]
        deg = torch.zeros(n, dtype=x.dtype, device=x.device)
        deg = deg.index_add(0, i, torch.ones_like(mu[i])).index_add(0, j, torch.ones_like(mu[j]))
        xm = 0.5 * (x[i] + x[j])
        v = step * Df / dr ** 2 * 0.5 * (M.beta[i] + M.beta[j]) * xm * (1 - xm) * (mu[i] - mu[j])
        keep = v.abs() >= min_dx
        i, j, v = i[keep], j[keep], v[keep]
        out, room = x / deg, torch.clamp(max_x - x, min=0.0) / deg
        hi, lo = torch.minimum(out[i], room[j]), -torch.minimum(out[j], room[i])
        return i, j, v, hi, lo

    for _ in range(nsteps):
        mu, act = potential()
        m = 1
        if control:
            i, j, v, hi, lo = moves(mu, act, dt)
            dx = zero.index_add(0, i, v).index_add(0, j, -v).abs().max() / max_dx
            over = torch.where((v > hi) & (hi > 0), v / hi, zero[:1])
            over = torch.maximum(over, torch.where((v < lo) & (lo < 0), v / lo, zero[:1]))
            need = max(float(dx), float(over.max()) if len(over) else 0.0)
            m = int(min(max_sub, max(1, math.ceil(need))))
        for k in range(m):
            if k:
                mu, act = potential()
            i, j, v, hi, lo = moves(mu, act, dt / m)
            v = torch.minimum(torch.maximum(v, lo), hi)
            x = x.index_add(0, i, -v).index_add(0, j, v)
    return dict(x=x.cpu().numpy(), mu=mu.cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("serve", "relax"):
        return None  # an optimiser's path: its steps hang on the ones before them
    if kind == "batch":
        return dict(totals=np.stack([_Model(s).evaluate()["totals"]
                                     for s in _batch_systems(case, seed)]))
    s = system(case, seed)
    if kind == "stretch":
        return _exact_stretch(s)
    if kind == "dmd":
        return _exact_dmd(s, case["nsteps"], case["control"]) \
            if len(s["x"]) * case["nsteps"] <= 450000 else None
    return _Model(s).evaluate()
