"""The edge audit's counting of an edge for two faces next to each other, its second
window, and the time of a fan, whose centre's window every spoke would ask."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def fan(n, hub=0):
    i = np.arange(n) + (hub == 0)
    i = i + (i >= hub) * (hub != 0)   # ids around the centre's
    return np.stack([np.full(n, hub), i, np.append(i[1:], i[-1] + 1 + (i[-1] + 1 == hub))], 1)


def strip(n):
    i = np.arange(n)
    return np.where((i % 2 == 0)[:, None], np.stack([i, i + 1, i + 2], 1), np.stack([i + 1, i, i + 2], 1))


def cases():
    rng = np.random.default_rng(4)
    for n in (1, 2, 31, 32, 33, 255, 256, 257, 5000):   # the ends of warps and blocks
        yield f"strip {n}", strip(n)
        yield f"soup {n}", np.arange(3 * n).reshape(n, 3)
    for k in (2, 3, 4, 5, 33):   # runs of equal edges over several lanes
        yield f"each face {k} times", np.repeat(strip(200), k, 0)
        yield f"one edge in {k} faces", np.stack([np.zeros(k), np.ones(k), np.arange(k) + 2], 1)
        yield f"every vertex order, {k}", np.concatenate([np.roll(strip(97), j % 3, 1)[:, ::1 - 2 * (j % 2)] for j in range(k)])
    for hub in (0, 2500, 5001):
        yield f"fan around {hub}", fan(5000, hub)
    yield "fans", np.concatenate([fan(100) + 101 * k for k in range(60)])
    yield "few ids", rng.integers(0, 4, (3000, 3))
    yield "degenerate", np.array([[0, 0, 1], [0, 0, 1], [1, 0, 0], [2, 2, 2], [2, 2, 2], [2, 0, 2]])
    # both windows of an edge fill up: complete bipartite hubs, and ids that share windows
    a, b = np.meshgrid(np.arange(40), 1000 + np.arange(40), indexing="ij")
    yield "two sets of hubs", np.stack([a.ravel(), b.ravel(), 5000 + np.arange(1600)], 1)
    yield "shared windows", np.stack([128 * np.arange(80), 128 * (100 + np.arange(80)), 128 * np.full(80, 300)], 1)


@pytest.mark.parametrize("name,faces", list(cases()), ids=[c[0] for c in cases()])
def test_counts(built, name, faces):
    import gpupr_capi

    F = np.ascontiguousarray(faces, np.int32)
    want = orc.edge_audit(F)
    for _ in range(3):
        assert gpupr_capi.edge_audit(F)[0] == want


def test_negative_index(built):
    import gpupr_capi

    F = strip(100).astype(np.int32)
    for at in (0, 31, 32, 99):
        for k in range(3):
            G = F.copy()
            G[at, k] = -1
            with pytest.raises(gpupr_capi.GpuprError, match="negative vertex index"):
                gpupr_capi.edge_audit(G)


def test_fan_takes_no_longer(built):
    """The edges of a fan of 4M faces are counted in less than twice the time of as
    many faces that share nothing (3 times, when each spoke asked the centre's
    whole window)."""
    import gpupr_capi

    n = 4_000_000
    i = torch.arange(n, device="cuda", dtype=torch.int32)
    fan = torch.stack([torch.zeros_like(i), i + 1, i + 2], 1).contiguous()
    soup = torch.arange(3 * n, device="cuda", dtype=torch.int32).view(n, 3)

    def ms(f):
        t = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            gpupr_capi.edge_audit(f)
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return sorted(t)[4]

    assert ms(fan) < 2 * ms(soup)
