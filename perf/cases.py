"""The calculations that programs give this framework, for measuring it.

A case is one call sequence of a host program on one GPU: a whole mg-manual
calculation (fill, solve, energy, the potential back in the caller's memory),
a focusing chain, a batch of ligands, a burst through the serving loop, a
solve on maps that the host filled, or a calculation with forces.  A program
keeps its calculation (the device arrays and captured graphs of one grid
shape) and pinned buffers for the results, so those are made in `prepare`;
everything from the atom arrays to the potential is in `run`.

Molecules are seeded globular clusters at the density of the benchmark's
(500 atoms in a 12 A ball, pairwise separation of at least 1.5 A, charges
from {-1, -1/2, 0, 1/2, 1}, radii 1.2-2.0 A), drawn in an ellipsoid with the
proportions of the grid, which leaves `margin` A around the molecule.

`exact` states the same calculations in 64-bit torch: the maps by the formulas
of the fill, the equation solved to rounding by conjugate gradients (and
Newton steps where it is nonlinear) instead of multigrid.
"""
import math

import numpy as np
import torch

from apbs_b200 import serve, synth
from apbs_b200.vpmg import FP64, MIXED, Vpmg, batch_solve

DIMES = (33, 49, 65, 97, 129, 161, 193, 225)
SURFACES = {"mol": synth.SRFM_MOL, "smol": synth.SRFM_SMOL, "spl2": synth.SRFM_SPL2}
BOUNDARIES = {"zero": synth.BCFL_ZERO, "sdh": synth.BCFL_SDH, "mdh": synth.BCFL_MDH}


def _case(kind, precision, dime, atoms, npbe=False, salt=0.1, valence=1, surface="smol",
          bcfl="sdh", net=0, margin=5.0, etol=0.0, count=1):
    nx, ny, nz = dime
    return dict(kind=kind, precision=precision, nx=nx, ny=ny, nz=nz, atoms=atoms, npbe=npbe,
                salt=salt, valence=valence, surface=surface, bcfl=bcfl, net=net, margin=margin,
                etol=etol, count=count)


def listed():
    return [
        # a ligand alone: the smallest calculation, all launches and latency
        dict(_case("solve", "fp64", (33, 33, 33), 40, salt=0.15, net=-1), name="ligand33_fp64"),
        # a peptide in mixed precision: an ordinary small request of a server
        dict(_case("solve", "mixed", (65, 65, 65), 500, salt=0.15), name="peptide65_mixed"),
        # an elongated protein, so a ragged grid; 2:1 salt, nonlinear, drop-in precision
        dict(_case("solve", "fp64", (97, 129, 65), 2217, npbe=True, valence=2, net=5,
                   surface="mol", bcfl="mdh"), name="elongated_fp64"),
        # the benchmark's calculation: a 5000-atom protein, nonlinear, both precisions
        dict(_case("solve", "mixed", (161, 161, 161), 5000, npbe=True, net=12),
             name="protein161_mixed"),
        dict(_case("solve", "fp64", (161, 161, 161), 5000, npbe=True, net=12),
             name="protein161_fp64"),
        # a receptor-ligand complex of a binding sweep, which solves to 1e-9
        dict(_case("solve", "mixed", (129, 129, 129), 3040, salt=0.15, net=-1, etol=1e-9),
             name="complex129_mixed"),
        # a large assembly, linear, drop-in precision: the largest grid served
        dict(_case("solve", "fp64", (225, 225, 225), 8000), name="assembly225_fp64"),
        # mg-auto style focusing: the whole protein at 97^3, then a site of it at 129^3
        dict(_case("focus", "fp64", (129, 129, 129), 5000, net=12), name="focus129_fp64"),
        # the free ligands of a binding sweep in one batch (33-65^3, to 1e-9)
        dict(_case("ligands", "mixed", (65, 65, 65), 40, salt=0.15, net=-1, etol=1e-9, count=16),
             name="ligands_mixed"),
        # spline surface and the forces on every atom, as a dynamics step asks for them
        dict(_case("forces", "fp64", (65, 97, 65), 700, salt=0.15, surface="spl2", margin=8.0),
             name="forces_fp64"),
        # the unchanged apbs program behind the drop-in: maps filled on the host
        dict(_case("maps", "fp64", (97, 97, 97), 1500), name="hostmaps97_fp64"),
        # requests of mixed sizes arriving together at the serving loop
        dict(_case("burst", "mixed", (129, 129, 129), 2500, count=16), name="burst_mixed"),
    ]


def draw(rng):
    kind = rng.choices(("solve", "focus", "ligands", "forces", "maps", "burst"),
                       (70, 7, 6, 6, 6, 5))[0]
    precision = rng.choice(("fp64", "mixed"))
    salt = 0.0 if rng.random() < 0.1 else round(rng.uniform(0.01, 0.3), 4)
    margin = round(rng.uniform(5.0, 12.0), 2)

    def atoms(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "ligands":
        return _case(kind, "mixed", (65, 65, 65), atoms(20, 200), salt=salt, net=-1,
                     margin=margin, etol=1e-9, count=rng.randint(2, 24))
    if kind == "burst":
        return _case(kind, precision, (129, 129, 129), atoms(300, 3000), salt=salt,
                     margin=margin, count=rng.randint(4, 16))
    if kind == "focus":
        n = rng.choice((97, 129, 161))
        return _case(kind, precision, (n, n, n), atoms(2000, 8000), salt=salt, margin=margin,
                     net=rng.randint(-10, 10))
    top = {"forces": 129, "maps": 161}.get(kind, 225)
    sizes = [n for n in DIMES if n <= top]
    n = rng.choice(sizes)
    dime = (n, n, n)
    if rng.random() < 0.4:  # an elongated or flat molecule
        near = [m for m in sizes if n / 2 < m < 2 * n]
        dime = (n, rng.choice(near), rng.choice(near))
    # as many atoms as give a spacing of about 0.3 to 1 A on this grid
    most = min(8000, max(60, int(500 * (max(min(dime) * 0.8 - 14, 6.0) / 24.0) ** 3)))
    least = max(20, int(500 * (max(min(dime) * 0.3 - 14, 0.0) / 24.0) ** 3))
    if kind == "forces":
        # the boundary forces want every atom's window inside the grid
        return _case(kind, precision, dime, atoms(least, max(least + 1, most // 2)), salt=salt,
                     surface="spl2", margin=margin + 3.0, npbe=rng.random() < 0.2)
    # the tight tolerance and the nonlinear equation where they are asked for
    npbe = kind == "solve" and rng.random() < 0.25 and (precision == "mixed" or max(dime) <= 161)
    tight = rng.random() < 0.3 and max(dime) <= 129
    return _case(kind, precision, dime, atoms(least, max(least + 1, most)), npbe=npbe, salt=salt,
                 valence=rng.choice((1, 1, 2)), surface=rng.choice(("smol", "smol", "mol")),
                 bcfl=rng.choice(("sdh", "sdh", "mdh", "zero")), net=rng.randint(-8, 12),
                 margin=margin, etol=1e-9 if tight else 0.0)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _molecule(atoms, dime, seed, net):
    """Random sequential packing of `atoms` points in an ellipsoid with the
    proportions of the grid and the benchmark molecules' density."""
    rng = np.random.default_rng(seed)
    n = np.asarray(dime, dtype=float) - 1.0
    axes = 12.0 * (atoms / 500.0) ** (1.0 / 3.0) * n / n.prod() ** (1.0 / 3.0)
    pts = np.empty((0, 3))
    while len(pts) < atoms:
        c = rng.uniform(-1.0, 1.0, (1024, 3))
        c = c[(c * c).sum(1) <= 1.0] * axes
        cell = np.floor(c / 8.0).astype(int)  # only points near a candidate can clash
        near = np.abs(c[:, None] - c[None]).max(2) < 1.5
        near &= ((c[:, None] - c[None]) ** 2).sum(2) < 1.5 ** 2
        ok = ~np.tril(near, -1).any(1)
        if len(pts):
            own = np.floor(pts / 8.0).astype(int)
            for key in np.unique(cell, axis=0):
                at = np.nonzero((cell == key).all(1) & ok)[0]
                by = pts[(np.abs(own - key) <= 1).all(1)]
                if len(at) and len(by):
                    ok[at] &= ((c[at][:, None] - by[None]) ** 2).sum(2).min(1) >= 1.5 ** 2
        pts = np.concatenate([pts, c[ok]])[:atoms]
    q = rng.choice([-1.0, -0.5, 0.0, 0.5, 1.0], size=atoms, p=[0.1, 0.2, 0.4, 0.2, 0.1])
    q += (net - q.sum()) / atoms
    shift = rng.uniform(-3.0, 3.0, 3)  # files have their molecules anywhere
    return synth.Molecule(pts + shift, q, rng.uniform(1.2, 2.0, atoms))


def _params(case, mol, dime=None, npbe=None, salt=None):
    dime = dime or (case["nx"], case["ny"], case["nz"])
    salt = case["salt"] if salt is None else salt
    z = case["valence"]
    ions = ((float(z), salt, 2.0), (-1.0, z * salt, 2.0)) if salt > 0 else ()
    span = mol.xyz.max(0) - mol.xyz.min(0) + 2 * 2.0 + 2 * case["margin"]
    p = synth.mg_manual(dime, tuple(span / (np.asarray(dime) - 1)), mol.center(),
                        npbe=case["npbe"] if npbe is None else npbe,
                        srfm=SURFACES[case["surface"]], bcfl=BOUNDARIES[case["bcfl"]], ions=ions,
                        etol=case["etol"])
    return p


def _jobs(case, seed):
    """The (params, molecule) pairs of one pass, from the seed alone."""
    dime = (case["nx"], case["ny"], case["nz"])
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "focus":
        mol = _molecule(case["atoms"], dime, seed, case["net"])
        ions = ((1.0, case["salt"], 2.0), (-1.0, case["salt"], 2.0)) if case["salt"] > 0 else ()
        span = float((mol.xyz.max(0) - mol.xyz.min(0)).max()) + 4.0 + 4 * case["margin"]
        pc, pf = synth.focus_pair(mol, 97, span / 96, case["nx"], 45.0 / (case["nx"] - 1),
                                  synth.subregion_center(mol, 30, seed + 100), ions=ions)
        return [(pc, mol), (pf, mol)]
    if case["kind"] == "ligands":
        out = []
        for k in range(case["count"]):
            n = (33, 49, 65)[k % 3]
            mol = _molecule(case["atoms"], (n, n, n), 1000 * seed + k, case["net"])
            out.append((_params(case, mol, (n, n, n)), mol))
        return out
    if case["kind"] == "burst":
        out = []
        for k in range(case["count"]):
            n = (65, 129, 33, 97)[k % 4]
            atoms = max(20, int(case["atoms"] * (n / 129.0) ** 2))
            mol = _molecule(atoms, (n, n, n), 1000 * seed + k, 0)
            out.append((_params(case, mol, (n, n, n), npbe=k % 5 == 4,
                                salt=case["salt"] * float(rng.uniform(0.1, 1.0))), mol))
        return out
    mol = _molecule(case["atoms"], dime, seed, case["net"])
    return [(_params(case, mol), mol)]


def _pinned(p):
    t = torch.empty((p.nz, p.ny, p.nx), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


class _State:
    """What the program keeps from one pass to the next."""

    def __init__(self, kind):
        self.kind = kind
        self.calcs, self.server = [], None

    def __del__(self):
        for c in self.calcs:
            c.close()
        if self.server is not None:
            self.server.close()


def prepare(case, seed):
    s = _State(case["kind"])
    precision = MIXED if case["precision"] == "mixed" else FP64
    s.jobs = _jobs(case, seed)
    s.u = [_pinned(p) for p, _ in s.jobs]
    if s.kind == "burst":
        s.server = serve.Server(precision=precision, max_inflight=8)
        return s
    s.calcs = [Vpmg(p, precision) for p, _ in s.jobs]
    if s.kind == "maps":
        # Vpmg_fillco on the host: here the device fill stands in for it once
        p, mol = s.jobs[0]
        with Vpmg(p, precision) as filler:
            filler.fillco(mol)
            m = filler.maps()
        s.maps = [m[k] for k in ("charge", "epsx", "epsy", "epsz", "kappa", "faces")]
    return s


def run(state):
    s = state
    if s.kind == "burst":
        ids = [s.server.submit(p, mol, u) for (p, mol), u in zip(s.jobs, s.u)]
        return {"energy": np.array([s.server.wait(i)["energy_kT"] for i in ids]), "u": s.u}
    if s.kind == "ligands":
        for c, (_, mol) in zip(s.calcs, s.jobs):
            c.fillco(mol)
        batch_solve(s.calcs)
        return {"energy": np.array([c.energy() for c in s.calcs]),
                "u": [c.potential_into(u) for c, u in zip(s.calcs, s.u)]}
    if s.kind == "focus":
        coarse, fine = s.calcs
        coarse.fillco(s.jobs[0][1])
        coarse.solve()
        fine.focus(coarse)
        fine.fillco(s.jobs[1][1])
        fine.solve()
        return {"energy": fine.energy(), "u": fine.potential_into(s.u[1])}
    calc = s.calcs[0]
    if s.kind == "maps":
        calc.set_coefficients(*s.maps)
    else:
        calc.fillco(s.jobs[0][1])
    calc.solve()
    out = {"energy": calc.energy(), "u": calc.potential_into(s.u[0])}
    if s.kind == "forces":
        out.update(calc.forces())
    return out


def _grids(case):
    """(points, atoms, nonlinear, potential wanted) of each grid of one pass."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "focus":
        return [(97 ** 3, case["atoms"], False, False), (n, case["atoms"], False, True)]
    if case["kind"] == "ligands":
        return [((33, 49, 65)[k % 3] ** 3, case["atoms"], False, True)
                for k in range(case["count"])]
    if case["kind"] == "burst":
        return [((65, 129, 33, 97)[k % 4] ** 3, case["atoms"], k % 5 == 4, True)
                for k in range(case["count"])]
    return [(n, case["atoms"], case["npbe"], True)]


def work(case):
    """Atoms (or maps) in, potentials out; and the arithmetic of the V-cycles
    that reduce the residual to the tolerance: about a decade each, 130
    operations per fine point and cycle (four smoothing sweeps, two residuals,
    the transfers, and a seventh more for the coarser levels), with one and a
    half times as many cycles for the nonlinear equation."""
    b = f = 0.0
    cycles = -math.log10(case["etol"] if case["etol"] > 0 else 1e-6)
    for n, atoms, npbe, out in _grids(case):
        b += 5 * 8 * n if case["kind"] == "maps" else 40 * atoms
        b += 8 * n if out else 0
        b += 72 * atoms if case["kind"] == "forces" else 0
        f += 130 * n * cycles * (1.5 if npbe else 1.0)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64-bit torch
# ---------------------------------------------------------------------------
class _Exact:
    """One calculation: maps, boundary values, potential, energy."""

    def __init__(self, p, mol):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.mol = p, mol
        self.n = (p.nx, p.ny, p.nz)
        self.h = (p.hx, p.hy, p.hz)
        self.lo = [p.center[d] - (self.n[d] - 1) * self.h[d] / 2.0 for d in range(3)]
        self.hi = [p.center[d] + (self.n[d] - 1) * self.h[d] / 2.0 for d in range(3)]
        self.xyz = self._t(mol.xyz)
        self.q, self.r = self._t(mol.charge), self._t(mol.radius)
        self.ions = [(p.ion_q[i], p.ion_conc[i], p.ion_radius[i]) for i in range(p.nion)]
        self.strength = sum(0.5 * c * z * z for z, c, _ in self.ions)
        self.rion = max([r for _, _, r in self.ions], default=0.0)
        na, ec, kb = 6.022045000e+23, 4.803242384e-10, 1.380662000e-16
        self.kappa2 = self.strength * 1e-16 * 8.0 * math.pi * na * ec * ec / (
            1000.0 * p.sdie * kb * p.temp)
        self.zmagic = 4.0 * math.pi * ec * ec / (kb * p.temp) * 1e8
        self._fill()

    def _t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)

    def _axis(self, d, shift=0.0):
        return self.lo[d] + shift + torch.arange(self.n[d], dtype=torch.float64,
                                                 device=self.dev) * self.h[d]

    def _cubes(self, pos, reach, shift):
        """Chunks of (rows, flat indices, squared distances per axis, on grid)
        of the grid points within `reach` of each position; the grid is
        shifted by half a spacing along the axes that `shift` marks."""
        rel = pos - self._t([self.lo[d] + (0.5 * self.h[d] if shift[d] else 0.0)
                             for d in range(3)])
        m = [int(math.ceil(2 * reach / self.h[d])) + 2 for d in range(3)]
        step = max(1, 8_000_000 // (m[0] * m[1] * m[2]))
        for a in range(0, len(pos), step):
            idx, d2, on = [], [], []
            for d in range(3):
                x = rel[a:a + step, d:d + 1]
                i = torch.floor((x - reach) / self.h[d]) + torch.arange(m[d], device=self.dev)
                t = x - self.h[d] * i
                idx.append(i.long())
                d2.append(t * t)
                on.append((i >= 0) & (i < self.n[d]))

            def cube(v, op):
                return op(op(v[2][:, :, None, None], v[1][:, None, :, None]),
                          v[0][:, None, None, :])
            flat = ((idx[2][:, :, None, None] * self.n[1] + idx[1][:, None, :, None]) * self.n[0]
                    + idx[0][:, None, None, :])
            yield slice(a, a + step), flat, cube(d2, torch.add), cube(on, torch.logical_and)

    def _mark(self, mask, pos, radius, value, shift=(0, 0, 0)):
        if not len(pos):
            return
        for rows, flat, d2, on in self._cubes(pos, float(radius.max()), shift):
            r = radius[rows][:, None, None, None]
            mask[flat[on & (d2 <= r * r)]] = value

    def _inside(self, pad):
        """Atoms within `pad` of the grid (strictly inside for pad 0)."""
        ok = torch.ones(len(self.xyz), dtype=torch.bool, device=self.dev)
        for d in range(3):
            x = self.xyz[:, d]
            ok &= (x > self.lo[d] - pad) & (x < self.hi[d] + pad)
        return ok

    def _surface_points(self):
        """Points of the solvent-accessible surface: each atom's inflated
        sphere, sampled, less the points inside another's."""
        p = self.p
        rmax = float(self.r.max()) + max(self.rion, p.srad) + 0.5
        npts = int(math.ceil(4.0 * math.pi * rmax * rmax * p.sdens))
        nth = int(math.floor(math.sqrt(math.pi * npts / 4.0) + 0.5))
        ref = []
        for it in range(nth):
            th = math.pi / nth * it
            nph = int(math.floor(math.sin(th) * 2 * nth + 0.5))
            for ip in range(nph):
                ph = 2 * math.pi / nph * ip
                ref.append((math.cos(ph) * math.sin(th), math.sin(ph) * math.sin(th),
                            math.cos(th)))
        ref = self._t(ref)
        ra = self.r + p.srad
        found = []
        for a in range(0, len(self.xyz), 32):
            x, rr = self.xyz[a:a + 32], ra[a:a + 32]
            gap = ((x[:, None] - self.xyz[None]) ** 2).sum(2)
            near = gap < (rr[:, None] + ra[None] + 1e-6) ** 2
            near[torch.arange(len(x)), torch.arange(a, a + len(x))] = False
            k = max(1, int(near.sum(1).max()))
            val, at = near.to(torch.int8).topk(k, dim=1)
            other, rad = self.xyz[at], torch.where(val > 0, ra[at], torch.zeros_like(ra[at]))
            pts = rr[:, None, None] * ref[None] + x[:, None]
            d2 = torch.zeros(len(x), len(ref), k, dtype=torch.float64, device=self.dev)
            for d in range(3):
                t = pts[:, :, None, d] - other[:, None, :, d]
                d2 += t * t
            found.append(pts[(d2 >= (rad * rad)[:, None]).all(2)])
        return torch.cat(found)

    def _fill(self):
        p, (nx, ny, nz) = self.p, self.n
        total, hv = nx * ny * nz, self.h[0] * self.h[1] * self.h[2]
        new = dict(dtype=torch.float64, device=self.dev)

        def bspline(x):
            lo = torch.where((x >= 0) & (x <= 2), 1 - (x - 1).abs(), torch.zeros_like(x))
            hi = torch.where((x >= 1) & (x <= 3), 1 - (x - 2).abs(), torch.zeros_like(x))
            s = 0.5 * x * lo + 0.5 * (3 - x) * hi
            return torch.where((x >= 0) & (x <= 3), s, torch.zeros_like(x))

        charge = torch.zeros(total, **new)
        idx, w = [], []
        for d in range(3):
            f = ((self.xyz[:, d] - self.lo[d]) / self.h[d])[:, None]
            i = torch.floor(f) - 1 + torch.arange(4, device=self.dev)
            on = (i >= 0) & (i < self.n[d])
            idx.append(i.long().clamp(0, self.n[d] - 1))
            w.append(torch.where(on, bspline(1.5 + (i - f)), torch.zeros_like(f)))
        flat = ((idx[2][:, :, None, None] * ny + idx[1][:, None, :, None]) * nx
                + idx[0][:, None, None, :])
        val = (self.q * self.zmagic / hv)[:, None, None, None] * w[0][:, None, None, :] * \
            w[1][:, None, :, None] * w[2][:, :, None, None]
        ok = torch.ones(len(self.xyz), dtype=torch.bool, device=self.dev)
        for d in range(3):
            ok &= (self.xyz[:, d] > self.lo[d] - self.h[d]) & (self.xyz[:, d] < self.hi[d] + self.h[d])
        charge.index_add_(0, flat[ok].reshape(-1), val[ok].reshape(-1))
        self.charge = charge.view(nz, ny, nx)

        half = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
        salt = 1.0 if self.strength > 0 else 0.0
        if p.srfm == synth.SRFM_SPL2:
            win = p.swin if p.swin > 0 else 0.3
            maps = []
            for shift, extra in (((0, 0, 0), self.rion),) + tuple((s, 0.0) for s in half):
                acc = torch.ones(total, **new)
                at = self._inside(0.0)
                pos, rad = self.xyz[at], self.r[at] + extra
                for rows, flat, d2, on in self._cubes(pos, float(rad.max()) + win, shift):
                    s = (d2.sqrt() - rad[rows][:, None, None, None] + win).clamp(0, 2 * win)
                    v = 0.75 * (s / win) ** 2 - 0.25 * (s / win) ** 3
                    on = on & (s < 2 * win)
                    acc.scatter_reduce_(0, flat[on], v[on], "prod")
                maps.append(acc.view(nz, ny, nx))
            self.kappa = salt * maps[0]
            self.eps = [(p.sdie - p.pdie) * m + p.pdie for m in maps[1:]]
        else:
            surf = self._surface_points()
            at = self._inside(0.0)
            eps = []
            for shift in half:
                m = torch.zeros(total, dtype=torch.bool, device=self.dev)
                self._mark(m, self.xyz[at], self.r[at] + p.srad, True, shift)
                self._mark(m, surf, torch.full((len(surf),), p.srad, **new), False, shift)
                eps.append(torch.where(m, p.pdie, p.sdie).to(torch.float64).view(nz, ny, nx))
            self.eps = self._smooth(eps) if p.srfm == synth.SRFM_SMOL else eps
            m = torch.full((total,), salt > 0, dtype=torch.bool, device=self.dev)
            if salt > 0:
                self._mark(m, self.xyz, self.r + self.rion, False)
            self.kappa = m.to(torch.float64).view(nz, ny, nx)

    def _smooth(self, eps):
        """Harmonic mean over a link's neighbours: itself, and the four links
        at each of its ends along the other two axes."""
        inv = [1.0 / e for e in eps]
        out = []
        for d in range(3):
            total, count = inv[d].clone(), torch.ones_like(inv[d])
            for o in range(3):
                if o == d:
                    continue
                for back in (0, 1):
                    for ahead in (0, 1):
                        src, dst = [slice(None)] * 3, [slice(None)] * 3
                        if ahead:
                            src[2 - d], dst[2 - d] = slice(1, None), slice(None, -1)
                        if back:
                            src[2 - o], dst[2 - o] = slice(None, -1), slice(1, None)
                        total[tuple(dst)] += inv[o][tuple(src)]
                        count[tuple(dst)] += 1
            out.append(count / total)
        return out

    # -- boundary values ----------------------------------------------------
    def _shell(self):
        """Indices (k, j, i) of the grid's outer points."""
        m = torch.ones(self.n[::-1], dtype=torch.bool, device=self.dev)
        m[1:-1, 1:-1, 1:-1] = False
        return m.nonzero(as_tuple=True)

    def boundary(self, coarse=None):
        u = torch.zeros(self.n[::-1], dtype=torch.float64, device=self.dev)
        if self.p.bcfl == synth.BCFL_ZERO:
            return u
        at = self._shell()
        x = [self._axis(d)[at[2 - d]] for d in range(3)]
        if coarse is not None:
            lo, fr = [], []
            for d in range(3):
                f = (x[d] - coarse.lo[d]) / coarse.h[d]
                i = torch.floor(f).clamp(0, coarse.n[d] - 2)
                lo.append(i.long())
                fr.append(f - i)
            v = torch.zeros_like(x[0])
            for c in range(8):
                b = [c & 1, c >> 1 & 1, c >> 2]
                wt = 1.0
                for d in range(3):
                    wt = wt * (fr[d] if b[d] else 1 - fr[d])
                v = v + wt * coarse.u[lo[2] + b[2], lo[1] + b[1], lo[0] + b[0]]
            u[at] = v
            return u
        p, kap = self.p, math.sqrt(self.kappa2)
        e, eps0, kb = 1.6021773e-19, 8.8541878e-12, 1.3806581e-23
        pre = e * e / (4 * math.pi * eps0 * kb * p.temp) * 1e10
        if p.bcfl == synth.BCFL_MDH:
            v = torch.zeros_like(x[0])
            step = max(1, 8_000_000 // len(v))
            for a in range(0, len(self.q), step):
                d2 = 0.0
                for d in range(3):
                    d2 = d2 + (x[d][:, None] - self.xyz[None, a:a + step, d]) ** 2
                dist, r = d2.sqrt(), self.r[a:a + step]
                v += (pre / p.sdie * self.q[a:a + step] / dist *
                      torch.exp(-kap * (dist - r)) / (1 + kap * r)).sum(1)
            u[at] = v
            return u
        mid = 0.5 * (self.xyz.max(0).values + self.xyz.min(0).values)
        rel = self.xyz - mid
        size = float((rel.pow(2).sum(1).sqrt() + self.r).max())
        mono, dip = self.q.sum(), (rel * self.q[:, None]).sum(0)
        quad = 1.5 * torch.einsum("a,ai,aj->ij", self.q, rel, rel)
        quad = (quad - torch.eye(3, dtype=torch.float64, device=self.dev) * quad.trace() / 3) / 3
        y = torch.stack([x[d] - mid[d] for d in range(3)], 1)
        dist = y.pow(2).sum(1).sqrt()
        er, ew = p.sdie / p.pdie, p.sdie
        t0, t1, t2 = 1 / ew / dist, -1 / ew / dist ** 3, 3 / ew / dist ** 5
        if kap < 1e-9:
            t1, t2 = 3 * er / (1 + 2 * er) * t1, 5 * er / (2 + 3 * er) * t2
        else:
            ka, kr = kap * size, kap * dist
            t0 = torch.exp(ka - kr) / (1 + ka) * t0
            t1 = 3 * er * torch.exp(ka - kr) * (1 + kr) * t1 / (
                1 + ka + er * (2 + 2 * ka + ka * ka))
            t2 = 5 * er * torch.exp(ka - kr) * (3 + 3 * kr + kr * kr) * t2 / (
                6 + 6 * ka + 2 * ka ** 2 + er * (9 + 9 * ka + 4 * ka ** 2 + ka ** 3))
        u[at] = pre * (mono * t0 - (y @ dip) * t1 + torch.einsum("ni,ij,nj->n", y, quad, y) * t2)
        return u

    # -- the equation -------------------------------------------------------
    def solve(self, coarse=None):
        h, hv = self.h, self.h[0] * self.h[1] * self.h[2]
        link = [self.eps[d] * (hv / h[d] ** 2) for d in range(3)]
        c = (slice(1, -1),) * 3

        def moved(d, s):
            t = [slice(1, -1)] * 3
            t[2 - d] = slice(2, None) if s > 0 else slice(None, -2)
            return tuple(t)
        up = [link[d][c].contiguous() for d in range(3)]
        dn = [link[d][moved(d, -1)].contiguous() for d in range(3)]
        diag = sum(up) + sum(dn)

        def couple(v):
            y = up[0] * v[moved(0, 1)]
            y.addcmul_(dn[0], v[moved(0, -1)])
            for d in (1, 2):
                y.addcmul_(up[d], v[moved(d, 1)]).addcmul_(dn[d], v[moved(d, -1)])
            return y

        def cg(dg, b, tol):
            x, full = torch.zeros_like(b), torch.zeros_like(self.charge)
            r, z = b.clone(), b / dg
            full[c] = z
            rz, stop = (r * z).sum(), tol * float(b.norm())
            for it in range(6000):
                pc = full[c]
                ap = dg * pc - couple(full)
                a = rz / (pc * ap).sum()
                x.addcmul_(pc, a)
                r.addcmul_(ap, -a)
                if it % 20 == 19 and float(r.norm()) <= stop:
                    break
                torch.div(r, dg, out=z)
                new = (r * z).sum()
                full[c] = z + (new / rz) * pc
                rz = new
            return x

        u = self.boundary(coarse)
        b = self.charge[c] * hv + couple(u)
        cc = self.p.sdie * self.kappa2 * self.kappa[c] * hv
        if not self.p.nonlin or not self.strength:
            x = torch.zeros_like(b)
            for _ in range(3):  # refined: the recurrence's residual drifts
                full = torch.zeros_like(u)
                full[c] = x
                x = x + cg(diag + cc, b - ((diag + cc) * x - couple(full)), 1e-9)
            u[c] = x
        else:
            w = [(-z, -0.5 / self.strength * n * z) for z, n, _ in self.ions]
            x, full = torch.zeros_like(b), torch.zeros_like(u)

            def residual(x):
                full[c] = x
                f = b + couple(full) - diag * x
                for z, s in w:
                    f = f - s * cc * torch.exp((z * x).clamp(-85, 85))
                return f
            f = residual(x)
            first = norm = float(f.norm())
            for _ in range(40):
                slope = sum(z * s * torch.exp((z * x).clamp(-85, 85)) for z, s in w) * cc
                step, damp = cg(diag + slope, f, 1e-4), 1.0
                while True:
                    trial = x + damp * step
                    g = residual(trial)
                    if float(g.norm()) < norm or damp < 1e-3:
                        break
                    damp *= 0.5
                x, f, norm = trial, g, float(g.norm())
                if norm <= 1e-13 * first:
                    break
            u[c] = x
        self.u = u
        return self

    # -- energy -------------------------------------------------------------
    def outside(self, fine):
        """Fixed-charge energy of the part of this grid outside a finer one."""
        w = []
        for d in range(3):
            x = self._axis(d)
            a = torch.maximum(x - self.h[d] / 2, torch.tensor(fine.lo[d], device=self.dev))
            b = torch.minimum(x + self.h[d] / 2, torch.tensor(fine.hi[d], device=self.dev))
            w.append(((b - a) / self.h[d]).clamp(0, 1))
        v = w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
        v = torch.where(v > 1e-9, torch.ones_like(v), v)
        return float(((1 - v) * self.u * self.charge).sum()) * math.prod(self.h) / self.zmagic

    def energy(self, outer=0.0):
        hv, u = math.prod(self.h), self.u
        qf = float((u * self.charge).sum()) * hv / self.zmagic + outer
        if not self.p.nonlin or not self.strength:
            return 0.5 * qf
        diel = 0.0
        c = (slice(None, -1),) * 3
        for d in range(3):
            t = [slice(None, -1)] * 3
            t[2 - d] = slice(1, None)
            diel += float((self.eps[d][c] * ((u[c] - u[tuple(t)]) / self.h[d]) ** 2).sum())
        qm = 0.0
        for z, n, _ in self.ions:
            qm += float((self.kappa * (torch.exp((-z * u).clamp(-85, 85)) - 1)).sum()) * n
        qm *= 0.5 * self.p.sdie * self.kappa2 / self.strength
        return qf - 0.5 * diel * hv / self.zmagic - qm * hv / self.zmagic


def exact(case, seed):
    jobs = _jobs(case, seed)
    if case["kind"] == "focus":
        coarse = _Exact(*jobs[0]).solve()
        fine = _Exact(*jobs[1]).solve(coarse)
        return {"energy": fine.energy(coarse.outside(fine)), "u": fine.u}
    energies, us = [], []
    for p, mol in jobs:
        e = _Exact(p, mol).solve()
        energies.append(e.energy())
        us.append(e.u.cpu().numpy())
    if case["kind"] in ("ligands", "burst"):
        return {"energy": np.array(energies), "u": us}
    out = {"energy": energies[0], "u": us[0]}
    if case["kind"] == "forces":  # only the potential behind them
        out.update(qf=None, db=None, ib=None)
    return out
