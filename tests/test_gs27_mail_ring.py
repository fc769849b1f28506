"""Host model of the mailbox wavefront (k_gs27_mail, apbs_b200/csrc/mg_kernels.cu):
every plane's CTA works on its own copies of planes k-1, k and k+1, and each
half-sweep goes through the plane's rows on its own.  Step j of half-sweep q
takes row j+1 of the lower plane's half-sweep q and row j+2 of the upper plane's
half-sweep q-1 from the inbox, updates row j from the three late neighbours
(lower plane (i, j+1), own plane (i+-1, j-1)) and the 23 others as they were at
the end of the step before, sends the row to the neighbour planes, and then reads
the early neighbours of row j+1.  It waits for half-sweep q-1 to have updated row
j+2 and for half-sweep q+1 to have entered step j - LAG; a loader fills the ring
of rows.

On adversarial interleavings of half-steps and loads the iterates equal the
sequential order's bit for bit, nothing deadlocks, an inbox ring of LAG + 2 rows
(8 at least) is never overwritten before it was taken, rows of x are loaded before
their owner stores them, and a ring slot is never refilled while its row is in
use.
"""
import random

import numpy as np
import pytest

OFFS = [(di, dj, dk) for dk in (-1, 0, 1) for dj in (-1, 0, 1) for di in (-1, 0, 1)
        if (di, dj, dk) != (0, 0, 0)]
LATE = {(0, 1, -1), (1, -1, 0), (-1, -1, 0)}
ROWS = 26  # rows of the ring at LAG <= 6


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
    def __init__(self, k, x, nhalf, rows):
        self.k, self.rows, self.loaded = k, rows, 3
        self.ring = {r: (r, x[k - 1:k + 2, r].copy()) for r in range(4)}
        self.inbox, self.early = {}, {}
        self.at = [-1] * nhalf     # the step each half-sweep is at
        self.half = [0] * nhalf    # 0: to take and update, 1: to read early neighbours
        self.prog = [-2] * nhalf

    def row(self, r):
        at, v = self.ring[r % self.rows]
        assert at == r, "row %d replaced by %d" % (r, at)
        return v


def run(x0, w, d, f, nhalf, fp, lag, pick):
    x = x0.copy()
    nz, ny, nx = x.shape
    irows = 8
    while irows < lag + 2:
        irows *= 2
    rows = max(ROWS, lag * (nhalf - 1) + 8)
    P = {k: Plane(k, x, nhalf, rows) for k in range(1, nz - 1)}

    def wants(p, q, j):
        if p.k > 1 and 0 <= j <= ny - 3:
            yield ("lo", q, j + 1)
        if p.k < nz - 2 and q > 0 and -1 <= j <= ny - 4:
            yield ("up", q - 1, j + 2)

    def ready(p, q):
        j = p.at[q]
        if j > ny - 1:
            return False
        if p.half[q] == 1:
            return True
        prep = 0 <= j <= ny - 3
        return (all(p.inbox.get((sd, n, r % irows), (None,))[0] == r for sd, n, r in wants(p, q, j))
                and p.loaded >= min(j + 2, ny - 1)
                and (q == 0 or not prep or p.prog[q - 1] >= min(j + 3, ny - 1))
                and (q + 1 == nhalf or p.prog[q + 1] >= j - lag))

    def send(p, q, j, vals):
        for side, kn in (("lo", p.k + 1), ("up", p.k - 1)):
            if kn < 1 or kn > nz - 2 or (side == "up" and q == nhalf - 1):
                continue
            box = P[kn].inbox
            key = (side, q, j % irows)
            assert key not in box, "inbox row overwritten"
            box[key] = (j, vals)

    def first_half(p, q):
        j = p.at[q]
        for sd, n, r in wants(p, q, j):
            for i, v in p.inbox.pop((sd, n, r % irows))[1]:
                p.row(r)[0 if sd == "lo" else 2, i] = v
        p.prog[q] = j
        if 1 <= j <= ny - 2:
            vals = []
            for i in colour(j, p.k, q, nx, fp):
                seen = p.early.pop((q, i))
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
            send(p, q, j, vals)

    def second_half(p, q):
        j = p.at[q] + 1
        if 1 <= j <= ny - 2:
            for i in colour(j, p.k, q, nx, fp):
                p.early[(q, i)] = {o: p.row(j + o[1])[1 + o[2], i + o[0]]
                                   for o in OFFS if o not in LATE}
        p.at[q] = j

    while True:
        todo = [(p, q) for p in P.values() for q in range(nhalf) if ready(p, q)]
        todo += [(p, -1) for p in P.values()
                 if p.loaded < ny - 1 and p.loaded + 1 <= p.prog[-1] + rows - 2]
        if not todo:
            assert all(min(p.at) == ny for p in P.values()), "deadlock"
            return x
        p, q = pick(todo)
        if q < 0:
            p.loaded += 1
            p.ring[p.loaded % rows] = (p.loaded, x[p.k - 1:p.k + 2, p.loaded].copy())
        elif p.half[q] == 0:
            first_half(p, q)
            p.half[q] = 1
        else:
            second_half(p, q)
            p.half[q] = 0


@pytest.mark.parametrize("nx,ny,nz", [(9, 9, 9), (7, 13, 11), (13, 5, 9), (5, 41, 7)])
@pytest.mark.parametrize("lag", [4, 6])
def test_mail_ring_equals_the_sequential_order(nx, ny, nz, lag):
    x0, w, d, f = make(nx, ny, nz, seed=nx * ny + nz + lag)
    for fp in (0, 1):
        want = sequential(x0, w, d, f, 4, fp)
        rng = random.Random(nx + 10 * ny + 100 * nz + lag)

        def step(t):
            p, q = t
            return p.at[q] if q >= 0 else p.loaded - 30

        for pick in (rng.choice, lambda r: max(r, key=step), lambda r: min(r, key=step),
                     lambda r: r[0], lambda r: r[-1],
                     lambda r: max(r, key=lambda t: (t[1], step(t))),
                     lambda r: min(r, key=lambda t: (t[1], step(t)))):
            assert np.array_equal(run(x0, w, d, f, 4, fp, lag, pick), want)
