"""CPU model of the dataflow factorization's schedule (k_chol_dataflow): the
tile ownership of dataflow_layout_t and the programs of the row, helper and
worker CTAs as coroutines that wait on the flags they poll on the device.
Every schedule must end with every tile published exactly once and its
updates applied in column order, whatever the order in which the CTAs run."""
import random

import pytest


def layout(nt, sms, row_tiles, helper_tiles):
    g = min(sms, nt * (nt + 1) // 2)
    dedicated = g >= 2 * nt
    rt = row_tiles if dedicated else 2
    ht = helper_tiles if g >= 4 * nt else 0
    rows, helpers = (nt if dedicated else 0), (nt if ht else 0)
    own = [[] for _ in range(g)]
    load = [0] * g
    for i in range(nt):
        for u in range(min(rt, i + 1)):
            own[i % g].append((i, i - u))
            load[i % g] += i - u + 1
        for u in range(rt, min(rt + ht, i + 1)):
            own[nt + i].append((i, i - u))
    first = rows + helpers
    for j in reversed(range(nt)):
        for i in range(j + rt + ht, nt):
            h = min(range(first, g), key=lambda c: load[c])
            own[h].append((i, j))
            load[h] += j + 1
    for o in own:
        o.sort(key=lambda t: (t[1], t[0]))
    return g, rows, helpers, own


class Run:
    def __init__(self, nt):
        self.nt, self.flags, self.y, self.k = nt, set(), set(), {}

    def update(self, t, k, *needs):
        assert all(f in self.flags for f in needs) and self.k.get(t, 0) == k, (t, k)
        self.k[t] = k + 1

    def publish(self, t):
        assert t not in self.flags and self.k.get(t, 0) == t[1], t
        self.flags.add(t)


def row_cta(r, i, tiles):
    t2 = (i, i - 2) if (i, i - 2) in tiles else None
    t1 = (i, i - 1) if i > 0 else None
    for k in range(max(0, i - 2 if t2 else i - 1)):
        need = [(i, k), (i - 1, k)] + ([(i - 2, k)] if t2 else [])
        while not (all(f in r.flags for f in need) and k in r.y):
            yield
        for t in filter(None, (t2, t1, (i, i))):
            r.update(t, k, (i, k))
    if t2:
        j = i - 2
        while (j, j) not in r.flags:
            yield
        r.publish(t2)
        while not ((i - 1, j) in r.flags and j in r.y):
            yield
        r.update((i, i), j, t2)
        r.update(t1, j, t2, (i - 1, j))
    if t1:
        while (i - 1, i - 1) not in r.flags:
            yield
        r.publish(t1)
        yield
        r.update((i, i), i - 1, t1)
        while i - 1 not in r.y:
            yield
    r.publish((i, i))
    yield
    r.y.add(i)


def helper_cta(r, i, tiles):
    c0, m = i - 2 - len(tiles), len(tiles)
    assert [t[1] for t in tiles] == list(range(c0, c0 + m))
    for k in range(c0):
        while not all(f in r.flags for f in [(i, k)] + [(c0 + u, k) for u in range(m)]):
            yield
        for u in range(m):
            r.update((i, c0 + u), k, (i, k), (c0 + u, k))
    for u in range(m):
        j = c0 + u
        while (j, j) not in r.flags:
            yield
        r.publish((i, j))
        while not all((j + v, j) in r.flags for v in range(1, m - u)):
            yield
        for v in range(1, m - u):
            r.update((i, j + v), j, (i, j), (j + v, j))


def worker(r, tiles):
    left = set(tiles)
    while left:
        for t in [t for t in tiles if t in left]:
            i, j = t
            k = r.k.get(t, 0)
            if k < j and (i, k) in r.flags and (j, k) in r.flags and (i != j or k in r.y):
                r.update(t, k, (i, k), (j, k))
                break
            if k == j and (i == j or (j, j) in r.flags):
                r.publish(t)
                left.discard(t)
                if i == j:
                    r.y.add(i)
                break
        yield


@pytest.mark.parametrize("row_tiles,helper_tiles", [(3, 3), (2, 0)])
@pytest.mark.parametrize("nt", [2, 3, 4, 5, 7, 9, 15, 37, 38, 39, 50, 76, 77, 90])
def test_every_schedule_ends(nt, row_tiles, helper_tiles):
    for seed in range(3):
        g, rows, helpers, own = layout(nt, 152, row_tiles, helper_tiles)
        assert sorted(t for o in own for t in o) == [(i, j) for i in range(nt) for j in range(i + 1)]
        r, ctas = Run(nt), []
        for c in range(g):
            if c < rows:
                ctas.append(row_cta(r, c, own[c]))
            elif c < rows + helpers:
                ctas.append(helper_cta(r, c - rows, own[c]))
            elif rows:   # two independent halves
                assert len(own[c]) <= 64
                ctas += [worker(r, own[c][0::2]), worker(r, own[c][1::2])]
            else:
                ctas.append(worker(r, own[c]))
        rng = random.Random(seed)
        for _ in range(40 * nt + 100):
            rng.shuffle(ctas)
            live = []
            for c in ctas:
                try:
                    next(c)
                    live.append(c)
                except StopIteration:
                    pass
            ctas = live
            if not ctas:
                break
        assert not ctas
        assert r.flags == {(i, j) for i in range(nt) for j in range(i + 1)} and len(r.y) == nt
