"""Surface validation accepts and refuses what a plain restatement of its rules does: triples distinct, in
range and not repeated, at most two faces per edge, one fan per vertex, no vertex without a face. Cases
around the per-vertex acceptance: open and closed fans, two fans at a vertex, hubs of 63 to 65 faces
and more, duplicates turned and flipped, and random soups."""
import numpy as np
import pytest

import rs_gb300 as R
from rs_gb300 import generators as gen


def valid(F, nv):
    F = np.asarray(F, int)
    if len({tuple(sorted(t)) for t in F}) != len(F) or any(len(set(t)) < 3 for t in F):
        return False
    edges = {}
    for f, t in enumerate(F):
        for k in range(3):
            edges.setdefault(frozenset((t[k], t[(k + 1) % 3])), []).append(f)
    if max(map(len, edges.values())) > 2:
        return False
    for v in range(nv):
        around = [f for f, t in enumerate(F) if v in t]
        if not around:
            return False
        seen, stack = {around[0]}, [around[0]]
        while stack:
            f = stack.pop()
            for u in F[f]:
                for g in edges.get(frozenset((v, u)), []) if u != v else []:
                    if g not in seen:
                        seen.add(g)
                        stack.append(g)
        if len(seen) != len(around):
            return False
    return True


def hub(m, closed):
    rim = np.arange(1, m + 1 if closed else m + 2)
    nxt = np.roll(rim, -1) if closed else rim[1:]
    return [[0, a, b] for a, b in zip(rim, nxt)], len(rim) + 1


def glued():  # two tetrahedra at one vertex
    t = [[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]]
    return t + [[0 if i == 0 else i + 3 for i in f] for f in t], 7


def cases():
    for m in (1, 2, 3, 63, 64, 65, 130):
        yield hub(m, False)
        if m > 2:
            yield hub(m, True)
    yield glued()
    P, F = gen.icosphere(1)
    F = F.astype(int)
    yield F, len(P)
    yield np.delete(F, [0, 7, 8], 0), len(P)                # open surfaces
    yield F, len(P) + 1                                     # a vertex without a face
    for t in (F[3], F[3][::-1], np.roll(F[3], 1)):
        yield np.vstack([F, t]), len(P)
    yield np.vstack([F, [F[0][0], F[0][1], len(P)]]), len(P) + 1   # three faces on an edge
    rng = np.random.default_rng(5)
    for i in range(300):
        nv = int(rng.integers(3, 8))
        n = int(rng.integers(1, 9))
        soup = np.array([rng.permutation(nv)[:3] for _ in range(n)])
        used = np.unique(soup)
        soup = np.searchsorted(used, soup)
        yield soup, len(used)
    for i in range(100):                                    # a sphere with a few faces left out or moved
        G = np.delete(F, rng.integers(0, len(F), rng.integers(0, 6)), 0)
        if i % 2:
            G[rng.integers(len(G))] = rng.permutation(len(P))[:3]
        yield G, len(P)


def test_validation_agrees_with_the_rules():
    rng = np.random.default_rng(1)
    accepted = 0
    for F, nv in cases():
        P = rng.standard_normal((nv, 3))
        ok = valid(F, nv)
        accepted += ok
        if ok:
            R.validate_surface(np.asarray(F, np.uint32), P)
        else:
            with pytest.raises(R.RsError):
                R.validate_surface(np.asarray(F, np.uint32), P)
    assert accepted > 60
