"""Staged host copies at the edges of their pieces and of the ring of staging
buffers, both directions, alone and from several threads."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


def roundtrip(rows, layout, seed):
    import gpupr_capi

    rng = np.random.default_rng(seed)
    a = rng.integers(-2**31, 2**31, (rows, 4), dtype=np.int64)
    if layout == "i4":
        a = a.astype(np.int32)
    elif layout == "f8":
        a = np.asfortranarray(a)
    out = torch.empty((rows, 4), dtype=torch.int32, device="cuda")
    gpupr_capi.upload_topology(a, out)
    torch.cuda.synchronize()
    return np.array_equal(out.cpu().numpy(), a.astype(np.int32))


@pytest.mark.parametrize("layout", ["i4", "i8", "f8"])
@pytest.mark.parametrize("nbytes", [16, MB - 16, MB, MB + 16, 4 * MB - 16, 4 * MB, 11 * MB, 32 * MB, 32 * MB + 16, 70 * MB + 48])
def test_upload(built, layout, nbytes):
    assert roundtrip(nbytes // 16, layout, nbytes)


def test_threads(built):
    ok = []
    t = [threading.Thread(target=lambda k=k: ok.append(roundtrip(3 * MB + k, ("i4", "f8")[k % 2], k))) for k in range(5)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert ok == [True] * 5


@pytest.mark.parametrize("n", [MB // 4 - 1, MB // 4, MB + 5, 9 * MB + 1])
def test_download(built, n):
    """Samples (4 bytes a tet) and labels to host arrays and to the device."""
    import gpupr_capi

    rng = np.random.default_rng(n)
    V = rng.random((1000, 3))
    T = rng.integers(0, 1000, (n, 4), dtype=np.int32)
    grid = dict(voxel_size=0.125, origin=np.zeros(3, np.int32), dims=np.ones(3, np.int32),
                background=np.float32(9.0), table=np.zeros((1, 1, 1), np.int32),
                values=rng.random((1, 8, 8, 8)).astype(np.float32))
    Vd, Td = torch.from_numpy(V).cuda(), torch.from_numpy(T).cuda()
    lab, s = gpupr_capi.sample_tet_labels(grid, V, T, (0, 0, 0), (1, 1, 1), 0.0, 0.5)
    lab_d, s_d = gpupr_capi.sample_tet_labels(grid, Vd, Td, (0, 0, 0), (1, 1, 1), 0.0, 0.5, device_out=True)
    assert np.array_equal(lab, lab_d.cpu().numpy()) and np.array_equal(s, s_d.cpu().numpy())
