"""Host model of the four-lane discharge (one lane an arc of a node): the split of
a node's excess over its admissible arcs by saturating 32-bit sums of the lanes
before, the relabel between steps, and the release of what was pushed.

Other blocks add to the node's excess while its four lanes load it.  One lane's
height, excess and terminal have to decide for all four: with a load of their own
each, lanes can split different amounts, and more or less is pushed than the
first lane releases, which makes or loses flow."""
from __future__ import annotations

import numpy as np
import pytest

U32 = 0xFFFFFFFF
UNVIS = U32


def discharge(h, ex, t, r, hn, n, local_steps):
    """h, ex, t as each of the four lanes knows them.  Returns what each arc and
    the sink got and what the first lane releases."""
    h, ex, t, r = list(h), list(ex), list(t), list(r)
    arcs, sink, pushed = [0] * 4, 0, [0] * 4
    live = [h[k] < n and ex[k] > 0 for k in range(4)]
    for step in range(local_steps):
        if not any(live):
            break
        for k in range(4):
            if live[k] and t[k] < 0 and h[k] == 1:
                x = min(ex[k], -t[k])
                t[k] += x
                ex[k] -= x
                pushed[k] += x
                sink += x if k == 0 else 0
        a = [r[k] if live[k] and hn[k] < h[k] else 0 for k in range(4)]
        x1 = [a[k ^ 1] for k in range(4)]
        p1 = [min(a[k] + x1[k], U32) for k in range(4)]
        x2 = [p1[k ^ 2] for k in range(4)]
        total = [min(p1[k] + x2[k], U32) for k in range(4)]
        for k in range(4):
            e = min(ex[k], U32) if ex[k] > 0 else 0
            before = min((x1[k] if k & 1 else 0) + (x2[k] if k & 2 else 0), U32)
            y = min(max(e - before, 0), a[k])
            arcs[k] += y
            r[k] -= y
            if live[k]:
                used = min(e, total[k])
                ex[k] -= used
                pushed[k] += used
        live = [live[k] and ex[k] > 0 for k in range(4)]
        low = min([hn[k] if r[k] else UNVIS for k in range(4)])
        for k in range(4):
            if live[k]:
                m = 0 if t[k] < 0 else low
                h[k] = UNVIS if m == UNVIS else m + 1
                live[k] = h[k] < n and step + 1 < local_steps
    return arcs, sink, pushed[0]


def node(rng):
    n = 1000
    h = int(rng.integers(1, 12))
    hn = [int(x) for x in rng.integers(1, 14, 4)]
    r = [int(x) for x in rng.choice([0, 1, 7, 1000, 2**31, U32], 4)]
    t = -int(rng.integers(0, 50)) if h == 1 else 0
    ex = int(rng.choice([1, 5, 1000, U32, U32 + 1, 2**40]))
    return n, h, hn, r, t, ex


@pytest.mark.parametrize("local_steps", [1, 2, 8, 32])
def test_one_lanes_values_conserve_flow(local_steps):
    rng = np.random.default_rng(local_steps)
    for _ in range(3000):
        n, h, hn, r, t, ex = node(rng)
        arcs, sink, released = discharge([h] * 4, [ex] * 4, [t] * 4, r, hn, n, local_steps)
        assert sum(arcs) + sink == released <= ex
        assert all(a <= c for a, c in zip(arcs, r))


def test_a_load_a_lane_makes_flow():
    """The case the broadcast is for: the excess grows between two lanes' loads."""
    arcs, sink, released = discharge([2] * 4, [5, 5, 9, 9], [0] * 4, [3, 3, 3, 3], [1] * 4, 100, 1)
    assert sum(arcs) + sink != released


def test_first_lane_decides():
    """push_relabel.cu's discharge_quad takes height, excess and terminal of a
    node from its first lane before any of them is used."""
    from conftest import PKG

    src = (PKG / "csrc" / "push_relabel.cu").read_text()
    body = src[src.index("void discharge_quad("):]
    body = body[:body.index("for (int step = 0;")]
    for x in "h", "ex":
        cast = body.index(f"{x} = __shfl_sync(0xffffffffu, {x}, first);")
        assert cast < body.index("bool live =")
    assert body.index("t = ldcg(g.term + v)") < body.index("t = __shfl_sync(0xffffffffu, t, first);")
