"""Tail steps of a relabel (block 0 alone for several levels, option bfs_tail_max)
beside the grid's other blocks, many times over: short steps in quick succession
are where a late block could miss a count."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import cached_graph, to_cuda
from test_gpu_sublevels import grid_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [1, 64, 1024])
def test_grids(built, tail):
    import gpupr_capi

    for seed, n in ((1, 500), (2, 20_000), (3, 300_000)):
        dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in grid_graph(n, np.random.default_rng(seed), 20, 50)]
        flow, part, _ = gpupr_capi.solve_ell(*dev)
        for k in range(60):
            f, p, st = gpupr_capi.solve_ell(*dev, opts=gpupr_capi.options(bfs_tail_max=tail, blocks_per_sm=1 + k % 4))
            assert f == flow and torch.equal(p, part)


def test_cuts(built):
    import gpupr_capi

    steps = 0
    for kind in ("lattice", "box", "torus"):
        g = cached_graph(kind, 3, 300_000)
        t, n = to_cuda(g["tets"], g["neighbors"])
        out, st = gpupr_capi.graph_cut(g["vertices"], t, n, g["labels"], 10.0)
        for k in range(60):
            o = gpupr_capi.options(bfs_tail_max=1024, work_relabel_factor=0.05 if k % 2 else 0)
            p, s2 = gpupr_capi.graph_cut(g["vertices"], t, n, g["labels"], 10.0, opts=o)
            assert np.array_equal(p, out) and s2["adjusted_flow"] == st["adjusted_flow"]
            steps += s2["bfs_tail_steps"]
    assert steps > 0
