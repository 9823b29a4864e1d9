"""The edge audit's probe sequences: windows that overflow (fans, vertices of
many edges, ids sharing a window), counts past three, the smallest meshes."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def fan(n):
    i = np.arange(1, n + 1)
    return np.stack([np.zeros(n), i, i + 1], 1)


def cases():
    rng = np.random.default_rng(2)
    yield "one face", np.array([[0, 1, 2]])
    yield "one face twice", np.array([[0, 1, 2], [2, 1, 0]])
    for n in (3, 7, 8, 9, 5000):
        yield f"fan {n}", fan(n)
    yield "closed fan", np.concatenate([fan(999), [[0, 1000, 1]]])
    for k in (1, 2, 3, 4, 9):
        yield f"fan x{k}", np.concatenate([fan(100)] * k)
    yield "random ids", rng.integers(0, 3000, (20_000, 3))
    yield "sparse ids", rng.integers(0, 2**31 - 1, (20_000, 3))
    # lower ids that share one of the 128 windows of the smallest table
    yield "one window", np.stack([128 * np.arange(85), np.full(85, 20_000), np.full(85, 20_001)], 1)
    yield "degenerate", np.array([[0, 0, 0], [0, 0, 1], [5, 5, 5], [5, 5, 5]])


@pytest.mark.parametrize("name,faces", list(cases()), ids=[c[0] for c in cases()])
def test_table(built, name, faces):
    import gpupr_capi

    F = np.ascontiguousarray(faces, np.int32)
    assert gpupr_capi.edge_audit(F)[0] == orc.edge_audit(F)
