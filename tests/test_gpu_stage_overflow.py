"""Sub-levels that put more nodes on a block's stage than its half (1024) holds:
what overflows goes straight to the next queue.

Forests make the overflow certain.  One tree has a root, 4 children, 12
grandchildren and ``fan`` leaves; there are 64 trees for each of the blocks
(one a multiprocessor), which is one pass of the first level.  Excess at the roots
and sinks at the leaves: a block discharges its 64 roots, 256 children, 768
grandchildren, and those make 64 * fan leaves active at once.  All of it is one
round where the leaves fit the half; the ones beyond it are the next round's.
The other way round, sinks at the roots, a relabel's first step labels the same
counts: one step where the leaves fit, two where not."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_sublevels import check

pytestmark = pytest.mark.gpu


def forest(trees, fan, to_leaves):
    """fan: leaves of each tree (array), at most 36."""
    n = 17 * trees + int(fan.sum())
    nbr = np.full((n, 4), -1, np.int32)
    cap = np.zeros((n, 4), np.uint32)
    t = np.arange(trees)
    top = [t, trees + np.arange(4 * trees), 5 * trees + np.arange(12 * trees)]
    leaf = np.arange(17 * trees, n)
    tree = np.repeat(t, fan)
    start = np.concatenate([[0], np.cumsum(fan)])[:-1]
    # a tree's leaves go round its 12 grandchildren, three of them at most
    idx = np.arange(n - 17 * trees) - start[tree]
    owner = 5 * trees + 12 * tree + idx % 12

    def link(parent, slot, child, c):
        nbr[parent, slot] = child
        nbr[child, 0] = parent
        cap[(parent, slot) if to_leaves else (child, 0)] = c

    below = np.zeros(n, np.int64)   # leaves below a node
    below[leaf] = 1
    np.add.at(below, owner, 1)
    np.add.at(below, trees + (top[2] - 5 * trees) // 3, below[top[2]])
    np.add.at(below, (top[1] - trees) // 4, below[top[1]])
    link((top[1] - trees) // 4, (top[1] - trees) % 4, top[1], below[top[1]])
    link(trees + (top[2] - 5 * trees) // 3, 1 + (top[2] - 5 * trees) % 3, top[2], below[top[2]])
    link(owner, 1 + idx // 12, leaf, 1)
    ends = np.zeros((2, n), np.uint32)
    ends[0 if to_leaves else 1][top[0]] = below[top[0]]
    ends[1 if to_leaves else 0][leaf] = 1
    return nbr, cap, ends[0], ends[1]


FANS = [15, 16, 17, 36, "mixed"]
OPTS = [dict(), dict(bfs_in_arc_masks=-1), dict(discharge_warp_aggregate=1)]


def fans(fan, trees):
    if fan == "mixed":   # 1024 leaves a block give or take
        return np.random.default_rng(5).integers(14, 18, trees, endpoint=True)
    return np.full(trees, fan)


@pytest.mark.parametrize("opt", OPTS)
@pytest.mark.parametrize("fan", FANS)
def test_discharge(built, fan, opt):
    trees = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    st = check(*forest(trees, fans(fan, trees), True), blocks_per_sm=1, **opt)
    assert st["solve_blocks_per_sm"] == 1
    if fan != "mixed":
        assert (st["rounds"] == 1) == (fan <= 16)


@pytest.mark.parametrize("opt", OPTS)
@pytest.mark.parametrize("fan", FANS)
def test_relabel(built, fan, opt):
    trees = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    st = check(*forest(trees, fans(fan, trees), False), blocks_per_sm=1, **opt)
    if fan != "mixed" and st["global_relabels"] <= 2:   # the last one labels nothing
        assert (sum(st["bfs_steps_by_frontier"]) == 1) == (fan <= 16)
