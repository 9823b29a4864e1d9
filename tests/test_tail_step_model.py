"""Host model of how the persistent solver's blocks agree on a BFS step when a tail
step (block 0 runs several levels alone) is among them: each block reads the
level's count from a ring of three, takes its branch, and meets the others at
grid barriers.  Blocks run in random order between barriers.  Block 0 rewrites
every counter of the ring and the level to go on from in its tail step, so all
blocks have to have read them before: without a barrier there, a block that comes
late reads a later count and leaves the others' path (on the GPU: a barrier that
never fills, or a queue read past its end)."""
from __future__ import annotations

import random

import pytest

BARRIER = object()


def block(b, ring, shared, counts, tail_max, tail_levels, before_tail, path):
    """One block's way through a relabel; counts[L] is level L's true frontier size."""
    level = 1
    for _ in range(4 * len(counts)):
        yield
        cnt = ring[level % 3]
        path.append((level, cnt))
        if cnt == 0:
            return
        if b == 0:
            ring[(level + 2) % 3] = 0
        if cnt <= tail_max:
            if before_tail:
                yield BARRIER
            if b == 0:
                at = level
                while True:
                    at += 1
                    yield
                    if counts[at] == 0 or counts[at] > tail_max or at - level >= tail_levels:
                        break
                ring[:] = [0, 0, 0]
                ring[at % 3] = counts[at]
                shared["level"] = at
            yield BARRIER
            yield
            level = shared["level"]
            continue
        yield
        if b == 0:
            ring[(level + 1) % 3] = counts[level + 1]
        yield BARRIER
        level += 1


def relabel(rng, before_tail, blocks=5):
    counts = [0] + [rng.choice((3, 5, 8, 100, 200)) for _ in range(rng.randint(2, 14))] + [0, 0, 0]
    ring, shared, paths = [0, counts[1], 0], {"level": 0}, [[] for _ in range(blocks)]
    runs = [block(b, ring, shared, counts, 10, rng.choice((1, 2, 5)), before_tail, paths[b]) for b in range(blocks)]
    state = ["run"] * blocks   # run, wait, done
    while any(s != "done" for s in state):
        ready = [b for b in range(blocks) if state[b] == "run"]
        if not ready:
            if any(s == "done" for s in state):
                return None   # some wait for blocks that have left
            state = ["run"] * blocks
            continue
        b = rng.choice(ready)
        try:
            state[b] = "wait" if next(runs[b]) is BARRIER else "run"
        except StopIteration:
            state[b] = "done"
    return paths


@pytest.mark.parametrize("seed", range(8))
def test_all_blocks_take_one_path(seed):
    rng = random.Random(seed)
    for _ in range(300):
        paths = relabel(rng, True)
        assert paths is not None and all(p == paths[0] for p in paths)


def test_a_late_block_leaves_it():
    rng = random.Random(1)
    runs = [relabel(rng, False) for _ in range(300)]
    assert any(p is None or any(q != p[0] for q in p) for p in runs)


def test_the_barrier_stands_before_the_tail():
    from conftest import PKG

    src = (PKG / "csrc" / "push_relabel.cu").read_text()
    body = src[src.index("cnt <= g.tail_max) {"):]
    body = body[:body.index("bfs_tail_body(")]
    assert "grid_barrier(" in body
