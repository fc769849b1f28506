"""Host model of the mailbox wavefront (k_gs27_mail, apbs_b200/csrc/mg_kernels.cu):
every plane's CTA works on its own copies of planes k-1, k and k+1; each
half-sweep has two groups, for the rows of either parity.  For row j a group
(1) takes row j+1 of the upper plane's half-sweep q-1 from the inbox, once the
other group took row j, half-sweep q-1 updated row j+1 and half-sweep q+1 row
j - LAG; (2) reads the neighbours that are not late; (3) takes row j+1 of the lower
plane's half-sweep q once the other group updated row j-1, updates row j from the
late neighbours (lower plane (i, j+1) and (i+-1, j), own plane (i+-1, j-1)) and
what it read in (2), and sends the row to the neighbour planes.  A loader fills the
ring of rows.

On adversarial interleavings of these parts the iterates equal the sequential
order's bit for bit, nothing deadlocks, an inbox ring of LAG - 1 rows is never
overwritten before it was taken, rows of x are loaded before their owner
stores them, and a ring slot is never refilled while its row is in use.
"""
import random

import numpy as np
import pytest

OFFS = [(di, dj, dk) for dk in (-1, 0, 1) for dj in (-1, 0, 1) for di in (-1, 0, 1)
        if (di, dj, dk) != (0, 0, 0)]
LATE = {(0, 1, -1), (1, 0, -1), (-1, 0, -1), (1, -1, 0), (-1, -1, 0)}


def colour(j, k, q, nx, fp):
    return [i for i in range(1, nx - 1) if ((i + j + k) & 1) == ((fp + q) & 1)]


def make(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((nz, ny, nx))
    x[1:-1, 1:-1, 1:-1] = rng.normal(size=(nz - 2, ny - 2, nx - 2))
    w = rng.uniform(-0.2, 0.2, size=(len(OFFS), nz, ny, nx))
    return x, w, rng.uniform(4.0, 6.0, size=(nz, ny, nx)), rng.normal(size=(nz, ny, nx))


def update(k, j, i, w, d, f, value):
    acc = 0.0
    for n, (di, dj, dk) in enumerate(OFFS):
        acc += w[n, k, j, i] * value(di, dj, dk)
    return (f[k, j, i] + acc) / d[k, j, i]


def sequential(x, w, d, f, nhalf, fp):
    x = x.copy()
    nz, ny, nx = x.shape
    for q in range(nhalf):
        for k in range(1, nz - 1):
            for j in range(1, ny - 1):
                for i in colour(j, k, q, nx, fp):
                    x[k, j, i] = update(k, j, i, w, d, f,
                                        lambda di, dj, dk: x[k + dk, j + dj, i + di])
    return x


class Plane:
    def __init__(self, k, x, nhalf, fp, rows):
        self.k, self.loaded, self.rows = k, 3, rows
        self.ring = {r: (r, x[k - 1:k + 2, r].copy()) for r in range(4)}
        self.inbox, self.early = {}, {}
        # per half-sweep and group (parity of row + plane colour): row, part
        self.group = {}
        for q in range(nhalf):
            for j in (0, 1):
                self.group[(q, self.of(q, j, fp))] = [j, 0]
        self.up = {g: -1 for g in self.group}
        self.done = {g: -1 for g in self.group}

    def of(self, q, j, fp):
        return ((1 + j + self.k) & 1) ^ ((fp + q) & 1)

    def row(self, r):
        at, v = self.ring[r % self.rows]
        assert at == r, "row %d replaced by %d" % (r, at)
        return v


def run(x0, w, d, f, nhalf, fp, lag, pick):
    x = x0.copy()
    nz, ny, nx = x.shape
    ROWS, IROWS = 3 * lag + 6, lag - 1  # rows of the ring and of the inbox
    P = {k: Plane(k, x, nhalf, fp, ROWS) for k in range(1, nz - 1)}

    def mail(p, side, q, j):
        return p.inbox.get((side, q, j % IROWS), (None,))[0] == j

    def has(p, side, q, j):  # row j + 1 comes by mail
        if j + 1 > ny - 2:
            return False
        return p.k > 1 if side == "lo" else (p.k < nz - 2 and q > 0)

    def ready(p, g):
        (q, b), (j, part) = g, p.group[g]
        inner = 1 <= j <= ny - 2
        if j > ny - 1:
            return False
        if part == 0:
            return ((not has(p, "up", q, j) or mail(p, "up", q - 1, j + 1))
                    and p.loaded >= min(j + 1, ny - 1) and p.up[(q, 1 - b)] >= j - 1
                    and (q == 0 or not inner or p.done[(q - 1, p.of(q - 1, j + 1, fp))] >= j + 1)
                    and (q + 1 == nhalf
                         or p.done[(q + 1, p.of(q + 1, j - lag, fp))] >= j - lag))
        if part == 1:
            return True
        return ((not has(p, "lo", q, j) or mail(p, "lo", q, j + 1))
                and p.done[(q, 1 - b)] >= j - 1)

    def take(p, side, q, j):
        for i, v in p.inbox.pop((side, q, j % IROWS))[1]:
            p.row(j)[0 if side == "lo" else 2, i] = v

    def advance(p, g):
        (q, b), (j, part) = g, p.group[g]
        inner = 1 <= j <= ny - 2
        if part == 0:
            if has(p, "up", q, j):
                take(p, "up", q - 1, j + 1)
            p.up[g] = j
        elif part == 1:
            if inner:
                p.early[g] = {i: {o: p.row(j + o[1])[1 + o[2], i + o[0]]
                                  for o in OFFS if o not in LATE}
                              for i in colour(j, p.k, q, nx, fp)}
        else:
            if has(p, "lo", q, j):
                take(p, "lo", q, j + 1)
            if inner:
                vals = []
                for i in colour(j, p.k, q, nx, fp):
                    seen = p.early[g][i]
                    vals.append((i, update(
                        p.k, j, i, w, d, f,
                        lambda di, dj, dk: p.row(j + dj)[1 + dk, i + di]
                        if (di, dj, dk) in LATE else seen[(di, dj, dk)])))
                for i, v in vals:
                    p.row(j)[1, i] = v
                    if q >= nhalf - 2:
                        for kn in (p.k - 1, p.k, p.k + 1):
                            assert kn not in P or P[kn].loaded >= j, "row stored before loaded"
                        x[p.k, j, i] = v
                for side, kn in (("lo", p.k + 1), ("up", p.k - 1)):
                    if 1 <= kn <= nz - 2 and not (side == "up" and q == nhalf - 1):
                        key = (side, q, j % IROWS)
                        assert key not in P[kn].inbox, "inbox row overwritten"
                        P[kn].inbox[key] = (j, vals)
            p.done[g] = j
        p.group[g] = [j, part + 1] if part < 2 else [j + 2, 0]

    while True:
        todo = [(p, g) for p in P.values() for g in p.group if ready(p, g)]
        todo += [(p, None) for p in P.values() if p.loaded < ny - 1 and p.loaded + 1 <=
                 min(p.done[(nhalf - 1, 0)], p.done[(nhalf - 1, 1)]) + ROWS - 2]
        if not todo:
            assert all(v[0] >= ny for p in P.values() for v in p.group.values()), "deadlock"
            return x
        p, g = pick(todo)
        if g is None:
            p.loaded += 1
            p.ring[p.loaded % ROWS] = (p.loaded, x[p.k - 1:p.k + 2, p.loaded].copy())
        else:
            advance(p, g)


@pytest.mark.parametrize("nx,ny,nz,lag", [(7, 7, 7, 4), (5, 21, 7, 4), (5, 13, 9, 5),
                                          (5, 41, 5, 8), (7, 5, 9, 11), (5, 61, 4, 14)])
def test_mail_ring_equals_the_sequential_order(nx, ny, nz, lag):
    x0, w, d, f = make(nx, ny, nz, seed=nx * ny + nz + lag)
    for fp in (0, 1):
        want = sequential(x0, w, d, f, 4, fp)
        rng = random.Random(nx + 10 * ny + 100 * nz + lag)

        def at(t):
            p, g = t
            return p.group[g][0] if g else p.loaded - 30

        def half(t):
            return t[1][0] if t[1] else -1

        for pick in (rng.choice, lambda r: max(r, key=at), lambda r: min(r, key=at),
                     lambda r: r[0], lambda r: r[-1],
                     lambda r: max(r, key=lambda t: (half(t), at(t))),
                     lambda r: min(r, key=lambda t: (half(t), at(t))),
                     lambda r: max(r, key=lambda t: (-half(t), at(t)))):
            assert np.array_equal(run(x0, w, d, f, 4, fp, lag, pick), want)
