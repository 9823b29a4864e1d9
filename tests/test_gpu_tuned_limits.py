"""A tuned size class changes the time of a solve, never whether it fits the
caller's limits: rounds that a small max_rounds or relabel period counts are as
long with an entry as without one, for a single solve and for a batch."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import cached_graph, to_cuda

pytestmark = pytest.mark.gpu
LIMITS = [(dict(max_rounds=16383), 8), (dict(global_relabel_period=63), 4), (dict(max_rounds=16383, global_relabel_period=63), 8)]


@pytest.fixture
def entries(built):
    """Entries for every size class, with a line and hops that no untuned solve uses."""
    import gpupr_capi

    old = gpupr_capi.tune_table(), gpupr_capi.batch_tune_table()

    def put(hops):
        t = [dict(size_class=k, blocks_per_sm=2, work_relabel_factor=1.0, solve_ms=1.0, default_ms=1.0,
                  chain_hops=hops, chain_max_active=hops) for k in range(32)] if hops else []
        gpupr_capi.set_tune_table(t)
        gpupr_capi.set_batch_tune_table(t)

    yield put
    gpupr_capi.set_tune_table(old[0])
    gpupr_capi.set_batch_tune_table(old[1])


@pytest.mark.parametrize("limit,levels", LIMITS)
@pytest.mark.parametrize("batch", [False, True])
def test_hops_under_limits(entries, limit, levels, batch):
    import gpupr_capi

    graphs = [cached_graph("torus", 5, 60_000), cached_graph("box", 4, 60_000)]
    toff, voff, V, T, Nb, L = gpupr_capi.pack_batch(graphs if batch else graphs[:1])
    t, n = to_cuda(T, Nb)

    def cut(**kw):
        o = gpupr_capi.options(**limit, **kw)
        if batch:
            out, _, st = gpupr_capi.graph_cut_batch(toff, voff, V, t, n, L, 10.0, opts=o)
        else:
            out, st = gpupr_capi.graph_cut(V, t, n, L, 10.0, opts=o)
        return np.asarray(out), (st["chain_hops"], st["chain_max_active"])

    entries(0)
    labels, short = cut()
    assert short == (levels, 131072)
    for tuned in 1, 4, 8, 40:
        entries(tuned)
        out, short = cut()
        assert short == (levels, 131072) and np.array_equal(out, labels)
        assert cut(chain_hops=7, chain_max_active=9)[1] == (7, 9)   # the caller's own count stands


def test_stats_report_what_ran(entries):
    """Short rounds run 16 sub-levels, or the hops asked for where that is more."""
    import gpupr_capi

    g = cached_graph("torus", 5, 60_000)
    t, n = to_cuda(g["tets"], g["neighbors"])

    def hops(**kw):
        return gpupr_capi.graph_cut(g["vertices"], t, n, g["labels"], 10.0, opts=gpupr_capi.options(**kw))[1]["chain_hops"]

    entries(0)
    assert [hops(), hops(chain_hops=1), hops(chain_hops=16), hops(chain_hops=40)] == [16, 16, 16, 40]
    entries(8)
    assert [hops(), hops(chain_hops=40)] == [16, 40]
    entries(0)
    e = gpupr_capi.autotune(g["vertices"], t, n, g["labels"], 10.0, reps=1)
    assert e["chain_hops"] == 16


@pytest.mark.parametrize("seed", [5, 6, 7])
def test_round_limits_that_held(built, seed):
    """A solve fits the round limits it fitted with chains of hops (63-92 rounds on
    these graphs; 207-265 with rounds of four sub-levels and 256 of them before a relabel)."""
    from test_gpu_sublevels import check, grid_graph

    g = grid_graph(200_000, np.random.default_rng(seed), 20, 50)
    for _ in range(3):
        assert check(*g, max_rounds=100)["rounds"] <= 100
