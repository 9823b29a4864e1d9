"""A batch's ranges of free nodes and its flows summed strip by strip, where
graph boundaries fall inside a warp's group of 128 nodes, on its edges, and
where strips hold several groups (above 1.2M free nodes): every graph's free
count, flows and labels must be those of its own cut (whole numbers, equal)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import cached_graph

pytestmark = pytest.mark.gpu


def with_free(g, count, rng):
    """g with `count` free tets (inner tets labelled 1 or 2), the rest 0."""
    inner = np.nonzero((g["neighbors"] >= 0).all(1))[0]
    lab = np.zeros(len(g["tets"]), np.uint8)
    pick = rng.choice(inner, size=count, replace=False)
    lab[pick] = rng.integers(1, 3, size=count)
    lab[(g["neighbors"] < 0).any(1)] = rng.integers(0, 2)
    return dict(g, labels=lab)


@pytest.mark.parametrize("counts,copies", [
    ([0, 1, 127, 128, 129, 0, 0, 31, 33, 96, 255, 256, 257, 1, 1, 1, 600, 0], 1),
    ([128] * 9, 3),
    ([3] * 300, 1),
    ([40_001, 5, 0, 39_990, 128], 20),
])
def test_free_ranges_and_flows_match_single_cuts(built, counts, copies):
    import gpupr_capi

    rng = np.random.default_rng(len(counts))
    small, large = cached_graph("proxy", 0, 6_000), cached_graph("box", 4, 60_000)
    graphs = [with_free(large if c > 1000 else small, c, rng) for c in counts]
    single = []
    for g in graphs:
        t, n = torch.from_numpy(g["tets"]).cuda(), torch.from_numpy(g["neighbors"]).cuda()
        single.append(gpupr_capi.graph_cut(g["vertices"], t, n, g["labels"], 10.0))
    toff, voff, V, T, Nb, L = gpupr_capi.pack_batch(graphs * copies)
    out, items, st = gpupr_capi.graph_cut_batch(toff, voff, V, torch.from_numpy(T).cuda(),
                                                torch.from_numpy(Nb).cuda(), L, 10.0)
    assert st["free_n"] == copies * sum(counts)
    for k, item in enumerate(items):
        lab, ost = single[k % len(graphs)]
        assert item["free_n"] == counts[k % len(graphs)], k
        assert item["raw_flow"] == ost["raw_flow"] and item["adjusted_flow"] == ost["adjusted_flow"], k
        assert np.array_equal(out[int(toff[k]):int(toff[k + 1])], lab), k
