"""Calls on the calling thread's own stream (cudaStreamPerThread, handle 2), whose
host arrays are large enough for helper threads to copy: the same handle in
another thread is another stream, so the copies have to be issued by the caller."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from conftest import cached_graph, to_cuda

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def own_stream(built, monkeypatch):
    import gpupr_capi

    def use(handle):
        torch.cuda.synchronize()
        monkeypatch.setattr(gpupr_capi, "_stream", lambda *a: ctypes.c_void_p(handle))

    yield use
    torch.cuda.synchronize()


@pytest.mark.parametrize("nbytes", [11 * MB, 70 * MB + 48])
@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("bits", [32, 64])
def test_upload(own_stream, nbytes, order, bits):
    import gpupr_capi

    a = np.random.default_rng(nbytes).integers(-2**31, 2**31, (nbytes // 16, 4), dtype=np.int64)
    a = np.asarray(a, np.int32 if bits == 32 else np.int64, order=order)
    out = torch.full(a.shape, -7, dtype=torch.int32, device="cuda")
    own_stream(2)
    gpupr_capi.upload_topology(a, out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), a.astype(np.int32))


def test_calls(own_stream):
    """A cut, a batch and a surface: everything from host arrays, the topology
    uploaded on the same stream just before, equal to an ordinary stream's."""
    import gpupr_capi

    g, h = cached_graph("box", 4, 900_000), cached_graph("torus", 5, 300_000)
    toff, voff, V, T, Nb, L = gpupr_capi.pack_batch([g, h])
    gt, gn, bt, bn = to_cuda(g["tets"], g["neighbors"], T, Nb)
    cut, st = gpupr_capi.graph_cut(g["vertices"], gt, gn, g["labels"], 10.0)
    batch, items, _ = gpupr_capi.graph_cut_batch(toff, voff, V, bt, bn, L, 10.0)
    SV, SF = gpupr_capi.surface(cut, g["vertices"], gt, gn)
    own_stream(2)
    for _ in range(3):
        t, n = torch.zeros_like(gt), torch.zeros_like(gn)
        torch.cuda.synchronize()
        gpupr_capi.upload_topology(np.asfortranarray(g["tets"].astype(np.int64)), t)
        gpupr_capi.upload_topology(g["neighbors"], n)
        out, st2 = gpupr_capi.graph_cut(g["vertices"], t, n, g["labels"], 10.0)
        assert np.array_equal(out, cut) and st2["adjusted_flow"] == st["adjusted_flow"]
        out, items2, _ = gpupr_capi.graph_cut_batch(toff, voff, V, bt, bn, L, 10.0)
        assert np.array_equal(out, batch)
        assert [i["adjusted_flow"] for i in items2] == [i["adjusted_flow"] for i in items]
        V2, F2 = gpupr_capi.surface(cut, g["vertices"], t, n)
        assert np.array_equal(F2, SF) and np.array_equal(V2, SV)
