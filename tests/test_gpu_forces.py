"""Per-atom forces (one CTA per atom) against numpy sums over the same maps
and potential: every term of Vpmg_qfForce (spl2 charges), Vpmg_dbForce and
Vpmg_ibForce with the cubic surface, added by numpy in its own order."""
import math

import numpy as np
import pytest

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, Vpmg

pytestmark = pytest.mark.gpu
WIN = 0.3


def _bspline(x):
    lo = np.where((x >= 0) & (x <= 2), 1 - np.abs(x - 1), 0.0)
    hi = np.where((x >= 1) & (x <= 3), 1 - np.abs(x - 2), 0.0)
    return np.where((x >= 0) & (x <= 3), 0.5 * x * lo + 0.5 * (3 - x) * hi, 0.0), lo - hi


def _grad(pos, center, arad):
    d = center - pos
    dist = np.sqrt((d * d).sum(-1))
    s = dist - arad + WIN
    on = (s > 1e-9) & (s < 2 * WIN - 1e-9)
    s = np.where(on, s, WIN)
    chi = 0.75 * s ** 2 / WIN ** 2 - 0.25 * s ** 3 / WIN ** 3
    dchi = 1.5 * s / WIN ** 2 - 0.75 * s ** 2 / WIN ** 3
    return np.where(on, -dchi / chi / np.maximum(dist, 1e-30), 0.0)[..., None] * d


def _forces(p, mol, u, maps):
    """(value, sum of |terms|) of qf, db, ib per atom."""
    h = np.array([p.hx, p.hy, p.hz])
    n = np.array([p.nx, p.ny, p.nz])
    lo = np.array([p.center[d] - (n[d] - 1) * h[d] / 2 for d in range(3)])
    hi = lo + (n - 1) * h
    strength = sum(0.5 * p.ion_conc[i] * p.ion_q[i] ** 2 for i in range(p.nion))
    pi, ec, kb, na = math.pi, 4.803242384e-10, 1.380662e-16, 6.022045e23
    zmagic = 4 * pi * ec * ec / (kb * p.temp) * 1e8
    zk2 = p.sdie * strength * 1e-16 * 8 * pi * na * ec * ec / (1000 * p.sdie * kb * p.temp)
    irad = max([p.ion_radius[i] for i in range(p.nion)], default=0.0)
    out = {k: np.zeros((mol.natoms, 2, 3)) for k in ("qf", "db", "ib")}
    eps = [maps["epsx"], maps["epsy"], maps["epsz"]]
    for a in range(mol.natoms):
        x, q, r = mol.xyz[a], mol.charge[a], mol.radius[a]
        f = (x - lo) / h
        if np.all((x > lo + h) & (x < hi - h)):
            i = np.floor(f).astype(int)[:, None] + np.arange(-1, 3)
            w, dw = _bspline(1.5 + i - f[:, None])
            v = u[np.ix_(i[2], i[1], i[0])]
            for d in range(3):
                k = [dw[e] if e == d else w[e] for e in range(3)]
                t = q * np.einsum("i,j,k,kji->kji", *k, v) / h[d]
                out["qf"][a, :, d] = t.sum(), np.abs(t).sum()
        rt = r + WIN + p.srad
        if np.all((x > lo + rt) & (x < hi - rt)):
            i0, i1 = np.floor((x - lo - rt) / h).astype(int), np.ceil((x - lo + rt) / h).astype(int)
            i = [np.arange(i0[d], i1[d] + 1) for d in range(3)]
            g = np.stack(np.meshgrid(*i, indexing="ij"), -1)
            at = (g[..., 2], g[..., 1], g[..., 0])
            t = np.zeros(g.shape)
            for d in range(3):
                for s in (1, -1):
                    e = np.zeros(3, int)
                    e[d] = 1
                    c = g + 0.5 * s * e
                    m = g if s > 0 else g - e
                    chi = (eps[d][m[..., 2], m[..., 1], m[..., 0]] - p.pdie) / (p.sdie - p.pdie)
                    nb = g + s * e
                    du = u[nb[..., 2], nb[..., 1], nb[..., 0]] - u[at]
                    t += _grad(x, lo + c * h, r) * (chi * du / h[d] ** 2)[..., None]
            t *= u[at][..., None] * -h.prod() * (p.sdie - p.pdie) * 0.5 / zmagic
            out["db"][a] = t.sum((0, 1, 2)), np.abs(t).sum((0, 1, 2))
        if zk2 > 0 and np.all((x > lo) & (x < hi)):
            rt = irad + r + WIN
            i = [np.arange(max(0, math.ceil(f[d] - rt / h[d])),
                           min(n[d] - 1, math.floor(f[d] + rt / h[d])) + 1) for d in range(3)]
            g = np.stack(np.meshgrid(*i, indexing="ij"), -1)
            at = (g[..., 2], g[..., 1], g[..., 0])
            uv, kv = u[at], maps["kappa"][at]
            if p.nonlin:
                mag = sum(kv * p.ion_conc[m] * (np.exp(np.clip(-p.ion_q[m] * uv, -85, 85)) - 1) / strength
                          for m in range(p.nion))
            else:
                mag = uv ** 2 * kv
            t = zk2 * mag[..., None] * _grad(x, lo + g * h, r + irad)
            t *= 0.5 * h.prod() / zmagic
            out["ib"][a] = t.sum((0, 1, 2)), np.abs(t).sum((0, 1, 2))
    return out


@pytest.mark.parametrize("natoms,dime,npbe", [(1, (33, 33, 33), False), (37, (33, 49, 33), True),
                                               (300, (65, 65, 65), False)])
def test_forces_match_numpy_sums(natoms, dime, npbe):
    mol = synth.cluster(natoms, 8.0 if natoms > 100 else 4.5, seed=natoms, net_charge=1.0)
    if natoms > 1:  # an atom within a spacing of the grid edge: no charge-field force
        mol.xyz[0] = mol.center() + np.array([0.5 * (dime[0] - 1) * 0.55 - 0.3, 0.0, 0.0])
    p = synth.mg_manual(dime, 0.55, mol.center() if natoms == 1 else mol.xyz[1:].mean(0),
                        npbe=npbe, srfm=synth.SRFM_SPL2,
                        ions=((1.0, 0.1, 2.0), (-1.0, 0.1, 2.0)))
    with Vpmg(p, FP64) as pmg:
        pmg.fillco(mol)
        pmg.solve()
        got, u, maps = pmg.forces(), pmg.u, pmg.maps()
    want = _forces(p, mol, u, maps)
    # two orders of one sum: at most its number of terms (under 1e5) roundings
    # of 1.1e-16, of the sum of the magnitudes; the terms themselves differ by
    # a few roundings of quotients whose distance to the window's end, down to
    # 1e-9 in extreme cases, is typically above 1e-3
    for k in ("qf", "db", "ib"):
        err = np.abs(got[k] - want[k][:, 0])
        assert np.all(err <= 1e-10 * (want[k][:, 1].max() + 1e-300)), k
    assert np.abs(got["db"]).max() > 0 and np.abs(got["ib"]).max() > 0
