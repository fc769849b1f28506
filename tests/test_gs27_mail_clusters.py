"""Host model of how the mailbox wavefront (k_gs27_mail,
apbs_b200/csrc/mg_kernels.cu) hands rows over: a row goes straight into the
inbox of a neighbour in the same cluster; for a foreign neighbour it goes to
the plane's global slots, and couriers of the neighbour's CTA move each
half-sweep's rows into its inbox in order.  The model has the waits of
tests/test_gs27_mail_ring.py without the values: on adversarial
interleavings every cluster size from one CTA to all the planes finishes
without overwriting an inbox row that was not taken, and couriers that serve
one side only do not finish in clusters of one CTA."""
import random

import pytest

NHALF = 4


def run(ny, nz, fp, lag, cluster, pick, both_sides=True):
    irows, last = lag - 1, nz - 2
    planes = range(1, last + 1)
    inbox = {k: {} for k in planes}   # (side, half-sweep, slot) -> row
    slots = set()                     # global: (plane, half-sweep, row)
    moved = {}                        # (plane, side, half-sweep) -> next row of its courier
    group = {}                        # (plane, half-sweep, group) -> [row, part]
    up, done = {}, {}

    def of(k, q, j):
        return ((1 + j + k) & 1) ^ ((fp + q) & 1)

    def foreign(k, n):
        return (k - 1) // cluster != (n - 1) // cluster

    for k in planes:
        for q in range(NHALF):
            for j in (0, 1):
                group[(k, q, of(k, q, j))] = [j, 0]
        sides = [(s, n) for s, n in (("lo", k - 1), ("up", k + 1)) if n in planes and foreign(k, n)]
        for s, n in sides if both_sides else sides[:1]:
            for q in range(NHALF - (s == "up")):
                moved[(k, s, q)] = 1
    for g in group:
        up[g] = done[g] = -1

    def put(k, side, q, j):
        key = (side, q, j % irows)
        assert key not in inbox[k], "inbox row overwritten"
        inbox[k][key] = j

    def has(k, side, q, j):  # row j + 1 comes by mail
        return j + 1 <= ny - 2 and (k > 1 if side == "lo" else k < last and q > 0)

    def there(k, side, q, j):
        return inbox[k].get((side, q, j % irows)) == j

    def ready(g):
        (k, q, b), (j, part) = g, group[g]
        if j > ny - 1:
            return False
        inner = 1 <= j <= ny - 2
        if part == 0:
            return ((not has(k, "up", q, j) or there(k, "up", q - 1, j + 1))
                    and up[(k, q, 1 - b)] >= j - 1
                    and (q == 0 or not inner or done[(k, q - 1, of(k, q - 1, j + 1))] >= j + 1)
                    and (q + 1 == NHALF or done[(k, q + 1, of(k, q + 1, j - lag))] >= j - lag))
        return ((not has(k, "lo", q, j) or there(k, "lo", q, j + 1))
                and done[(k, q, 1 - b)] >= j - 1)

    def advance(g):
        (k, q, b), (j, part) = g, group[g]
        if part == 0:
            if has(k, "up", q, j):
                del inbox[k][("up", q - 1, (j + 1) % irows)]
            up[g] = j
            group[g] = [j, 1]
            return
        if has(k, "lo", q, j):
            del inbox[k][("lo", q, (j + 1) % irows)]
        if 1 <= j <= ny - 2:
            for side, n in (("lo", k + 1), ("up", k - 1)):
                if n not in planes or (side == "up" and q == NHALF - 1):
                    continue
                if foreign(k, n):
                    slots.add((k, q, j))
                else:
                    put(n, side, q, j)
        done[g] = j
        group[g] = [j + 2, 0]

    while True:
        todo = [g for g in group if ready(g)]
        todo += [c for c, j in moved.items()
                 if (c[0] - 1 if c[1] == "lo" else c[0] + 1, c[2], j) in slots]
        if not todo:
            return all(j >= ny for j, _ in group.values())
        t = pick(todo)
        if t in group:
            advance(t)
        else:
            put(*t, moved[t])
            moved[t] += 1


def picks(seed):
    rng = random.Random(seed)

    def courier(t):
        return isinstance(t[1], str)

    return (rng.choice, lambda r: r[0], lambda r: r[-1],
            lambda r: min(r, key=lambda t: (courier(t), t[0])),
            lambda r: max(r, key=lambda t: (courier(t), t[0])),
            lambda r: max(r, key=lambda t: (courier(t), -t[0])))


@pytest.mark.parametrize("cluster", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("ny,nz,lag", [(9, 9, 6), (33, 7, 14), (13, 19, 4)])
def test_every_cluster_size_finishes(ny, nz, lag, cluster):
    for fp in (0, 1):
        for pick in picks(ny + nz + cluster):
            assert run(ny, nz, fp, lag, cluster, pick)


def test_couriers_of_one_side_would_hang_in_clusters_of_one():
    for pick in picks(1):
        assert not run(9, 9, 1, 6, 1, pick, both_sides=False)
        assert run(9, 9, 1, 6, 2, pick, both_sides=False)
