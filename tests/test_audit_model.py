"""Host model of how the edge audit shares equal edges between neighbouring lanes
of a warp: a lane counts an edge for itself and the next lane, unless the lane
before has that edge too.  Every edge of every face has to be counted once."""
from __future__ import annotations

import numpy as np
import pytest


def shared(E):
    """E[lane][k]: the edges of a warp's faces.  Returns how often each is counted."""
    n = len(E)
    to = [[None] * 3 for _ in range(n)]
    seen = [[False] * 3 for _ in range(n)]
    for l in range(n - 1):
        for j in range(3):
            for k in range(3):
                if E[l + 1][j] == E[l][k] and to[l][k] is None and not seen[l][j]:
                    to[l][k] = j
                    seen[l][j] = True
    c = [[1] * 3 for _ in range(n)]
    for l in range(n):
        before = seen[l - 1] if l else [False] * 3
        for k in range(3):
            if to[l][k] is not None and not before[k]:
                c[l][k] += 1
                c[l + 1][to[l][k]] -= 1
    return c


@pytest.mark.parametrize("ids", [2, 3, 5, 9, 1000])
def test_each_edge_once(ids):
    rng = np.random.default_rng(ids)
    for _ in range(400):
        F = rng.integers(0, ids, (32, 3))
        if rng.random() < 0.3:
            F = np.repeat(F[:11], 3, 0)[:32]
        E = [[tuple(sorted((f[k], f[(k + 1) % 3]))) for k in range(3)] for f in F]
        c = shared(E)
        assert all(0 <= x <= 2 for l in c for x in l)
        got, want = {}, {}
        for l in range(32):
            for k in range(3):
                got[E[l][k]] = got.get(E[l][k], 0) + c[l][k]
                want[E[l][k]] = want.get(E[l][k], 0) + 1
        assert got == want


def test_a_strip_shares_one_edge_a_face():
    F = [(i, i + 1, i + 2) for i in range(32)]
    E = [[tuple(sorted((f[k], f[(k + 1) % 3]))) for k in range(3)] for f in F]
    c = shared(E)
    assert sum(x == 2 for l in c for x in l) == 31
