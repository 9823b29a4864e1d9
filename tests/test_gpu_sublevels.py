"""The persistent solver's block sub-levels and four-lane discharge and BFS
steps, at the sizes and capacities where they can go wrong: graphs of a few
nodes up to several passes of a block, excess sums above 32 bits, short and
long local step counts, one block per SM (stage overflow).  Flow and partition
are whole numbers and must equal the exact CPU max flow's."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def grid_graph(n, rng, cap_hi, src_hi):
    """Four-neighbour rows on a near-square grid of n nodes, random integer
    capacities and terminals."""
    w = max(1, int(np.sqrt(n)))
    i = np.arange(n)
    nbr = np.full((n, 4), -1, np.int64)
    right = (i % w != w - 1) & (i + 1 < n)
    nbr[right, 0] = i[right] + 1
    left = i % w != 0
    nbr[left, 1] = i[left] - 1
    down = i + w < n
    nbr[down, 2] = i[down] + w
    up = i >= w
    nbr[up, 3] = i[up] - w
    cap = rng.integers(0, cap_hi, (n, 4), endpoint=True)
    cap[rng.random((n, 4)) < 0.2] = 0
    cap[nbr < 0] = 0
    src = np.where(rng.random(n) < 0.3, rng.integers(0, src_hi, n, endpoint=True), 0)
    snk = np.where(rng.random(n) < 0.1, rng.integers(0, src_hi, n, endpoint=True), 0)
    return nbr.astype(np.int32), cap.astype(np.uint32), src.astype(np.uint32), snk.astype(np.uint32)


def check(nbr, cap, src, snk, **kw):
    import gpupr_capi

    term = (src.astype(np.int64) - snk.astype(np.int64)).astype(np.int32)
    base = int(np.minimum(src, snk).astype(np.int64).sum())
    f, _, _, p = orc.maxflow_bk(nbr, cap, term)
    dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in (nbr, cap, src, snk)]
    flow, part, st = gpupr_capi.solve_ell(*dev, opts=gpupr_capi.options(**kw))
    assert flow == f + base
    assert np.array_equal(part.cpu().numpy(), p)
    return st


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 63, 64, 65, 257, 1025, 40_000])
def test_sizes(built, n):
    check(*grid_graph(n, np.random.default_rng(n), 20, 50))


@pytest.mark.parametrize("opt", [dict(), dict(local_steps=1), dict(local_steps=32), dict(blocks_per_sm=1),
                                 dict(bfs_in_arc_masks=-1), dict(max_rounds=16383), dict(max_rounds=16384),
                                 dict(chain_max_active=1), dict(chain_hops=4)])
@pytest.mark.parametrize("cap_hi,src_hi", [(3, 40), (0x7FFFFFFF, 0x7FFFFFFF)])
def test_wide_sums(built, opt, cap_hi, src_hi):
    """Capacities up to 2^31 - 1: four of them exceed 32 bits at a node."""
    check(*grid_graph(20_000, np.random.default_rng(7), cap_hi, src_hi), **opt)


def test_stage_overflow(built):
    """One block per SM and every node active: sub-levels of more nodes than a
    stage half holds."""
    check(*grid_graph(900_000, np.random.default_rng(3), 30, 9), blocks_per_sm=1, chain_max_active=1 << 30)


def test_round_limit(built):
    import gpupr_capi

    g = grid_graph(40_000, np.random.default_rng(5), 20, 50)
    with pytest.raises(gpupr_capi.GpuprError, match="max macro rounds"):
        check(*g, max_rounds=1)
