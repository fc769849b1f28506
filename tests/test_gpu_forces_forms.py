"""The other forms of the per-atom forces (one CTA per atom, k_forces) against numpy
sums: trilinear and 5th-order B-spline charges (qfForceSpline1, qfForceSpline4), and the
5th- and 7th-order window polynomials of srfm spl3 and spl4 in the boundary forces,
whose points the kernel picks by their distance to the atom's shell."""
import itertools
import math

import numpy as np
import pytest
import test_gpu_forces as base

from apbs_b200 import synth
from apbs_b200.vpmg import FP64, Vpmg

pytestmark = pytest.mark.gpu
WIN = base.WIN


def _poly(order, arad):
    """Window polynomial from 0 at arad - WIN to 1 at arad + WIN."""
    b, e = arad - WIN, arad + WIN
    if order == 3:
        d = math.pow(e - b, 5.0)
        e2, b2 = e * e, b * b
        b3 = b2 * b
        b4 = b3 * b
        return [(-10.0 * e2 * b3 + 5.0 * e * b4 - b4 * b) / d, (30.0 * e2 * b2) / d,
                (-30.0 * (e2 * b + e * b2)) / d, (10.0 * (e2 + 4.0 * e * b + b2)) / d,
                (-15.0 * (e + b)) / d, 6.0 / d]
    E, B = [1.0], [1.0]
    for _ in range(7):
        E.append(E[-1] * e)
        B.append(B[-1] * b)
    d = (E[7] - 7.0 * b * E[6] + 21.0 * B[2] * E[5] - 35.0 * E[4] * B[3] + 35.0 * E[3] * B[4] -
         21.0 * B[5] * E[2] + 7.0 * e * B[6] - B[7])
    return [B[4] * (35.0 * E[3] - 21.0 * b * E[2] + 7 * e * B[2] - B[3]) / d,
            -140.0 * B[3] * E[3] / d, 210.0 * E[2] * B[2] * (e + b) / d,
            -140.0 * e * b * (E[2] + 3.0 * b * e + B[2]) / d,
            35.0 * (E[3] + 9.0 * b * E[2] + 9.0 * e * B[2] + B[3]) / d,
            -84.0 * (E[2] + 3.0 * b * e + B[2]) / d, 70.0 * (e + b) / d, -20.0 / d]


def _grad(order):
    def grad(pos, center, arad):
        c = _poly(order, arad)
        d = center - pos
        dist = np.sqrt((d * d).sum(-1))
        on = (dist >= arad - WIN) & (dist <= arad + WIN) & \
            (np.abs(dist - (arad - WIN)) >= 1e-9) & (np.abs(dist - (arad + WIN)) >= 1e-9)
        s = np.where(on, dist, arad)
        powers = [np.ones_like(s)]
        for _ in c[1:]:
            powers.append(powers[-1] * s)
        chi, dchi = c[0] + c[1] * s, c[1]
        for k in range(2, len(c)):
            chi = chi + c[k] * powers[k]
            dchi = dchi + k * c[k] * powers[k - 1]
        on &= chi > 0.0
        chi = np.minimum(np.where(on, chi, 1.0), 1.0)
        return np.where(on, -(dchi / chi), 0.0)[..., None] * (d / np.where(on, dist, 1.0)[..., None])
    return grad


def _bspline4(x):
    """Centred quartic B-spline on (0, 5) and its derivative, from truncated powers."""
    sign = [1, -5, 10, -10, 5, -1]
    v = sum(s * np.maximum(x - k, 0.0) ** 4 for k, s in enumerate(sign)) / 24
    dv = sum(s * np.maximum(x - k, 0.0) ** 3 for k, s in enumerate(sign)) / 6
    return v, dv


def _charge_forces(chgm, p, mol, u):
    h = np.array([p.hx, p.hy, p.hz])
    n = np.array([p.nx, p.ny, p.nz])
    lo = np.array([p.center[d] - (n[d] - 1) * h[d] / 2 for d in range(3)])
    hi = lo + (n - 1) * h
    out = np.zeros((mol.natoms, 2, 3))
    for a in range(mol.natoms):
        x, q = mol.xyz[a], mol.charge[a]
        f = (x - lo) / h
        edge = 2 * h if chgm == synth.CHGM_SPL4 else 0 * h
        if not np.all((x > lo + edge) & (x < hi - edge)):
            continue
        if chgm == synth.CHGM_SPL4:
            i = np.floor(f).astype(int)[:, None] + np.arange(-2, 4)
            w, dw = _bspline4(2.5 + i - f[:, None])
            v = u[np.ix_(i[2], i[1], i[0])]
            for d in range(3):
                k = [dw[e] if e == d else w[e] for e in range(3)]
                t = q * np.einsum("i,j,k,kji->kji", *k, v) / h[d]
                out[a, :, d] = t.sum(), np.abs(t).sum()
        else:
            i0 = np.floor(f).astype(int)
            w = np.stack([1 - (f - i0), f - i0])
            for d in range(3):
                t = [-q * math.prod(2 * c[e] - 1 if e == d else w[c[e], e] for e in range(3)) *
                     u[i0[2] + c[2], i0[1] + c[1], i0[0] + c[0]] / h[d]
                     for c in itertools.product((0, 1), repeat=3)]
                out[a, :, d] = sum(t), sum(map(abs, t))
    return out


@pytest.mark.parametrize("chgm,order,npbe", [(synth.CHGM_TRIL, 3, False),
                                             (synth.CHGM_SPL4, 4, True),
                                             (synth.CHGM_SPL4, 3, False)])
def test_other_charges_and_surfaces_match_numpy(monkeypatch, chgm, order, npbe):
    mol = synth.cluster(40, 4.5, seed=9 + order, net_charge=1.0)
    mol.xyz[0] = mol.center() + np.array([8.4, 0.0, 0.0])  # near an edge of the grid
    p = synth.mg_manual((33, 49, 33), 0.55, mol.xyz[1:].mean(0), npbe=npbe,
                        srfm=synth.SRFM_SPL3 if order == 3 else synth.SRFM_SPL4,
                        ions=((1.0, 0.1, 2.0), (-1.0, 0.1, 2.0)))
    p.chgm = chgm
    with Vpmg(p, FP64) as pmg:
        pmg.fillco(mol)
        pmg.solve()
        got, u, maps = pmg.forces(), pmg.u, pmg.maps()
    monkeypatch.setattr(base, "_grad", _grad(order))
    want = base._forces(p, mol, u, maps)
    want["qf"] = _charge_forces(chgm, p, mol, u)
    # two orders of one sum of under 1e5 terms, as in test_gpu_forces; the terms' own
    # quotients lose digits where the window's polynomial is small: its coefficients
    # (up to 1e4 of its value at the shell) leave 1e-12 of a value above 1e-3, and the
    # terms below that are no larger than the window's others by more than 1e3
    for k in ("qf", "db", "ib"):
        err = np.abs(got[k] - want[k][:, 0])
        assert np.all(err <= 1e-8 * (want[k][:, 1].max() + 1e-300)), k
        assert np.abs(got[k]).max() > 0, k
