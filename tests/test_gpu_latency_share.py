"""Option latency_share: per mille of the batch's modelled time that a pair's
own latency may take; 60 is the default, and a smaller share favours the
classes that finish a pair sooner."""
import numpy as np
import pytest

import ipuma_b200 as ib
import workloads

pytestmark = pytest.mark.gpu


def _cells_by_kind(wl, share):
    with ib.Engine(ib.sw_config(wl.gap_init, wl.gap_extend, wl.match, wl.mismatch, wl.ambiguity, wl.similarity,
                                wl.datatype), ib.algo_config(forward_only=True)) as e:
        e.set_option("autotune", 0)
        e.set_option("time_launches", 1)
        if share:
            e.set_option("latency_share", share)
        got = e.compare(wl.codes, ib.make_pairs(wl.a_off, wl.a_len, wl.b_off, wl.b_len))
        st = e.stats()
    cells = {}
    for k in range(st.n_timed):
        cells[st.timed_kind[k]] = cells.get(st.timed_kind[k], 0) + st.timed_cells[k]
    return got, cells


def test_share_is_per_mille_of_the_batch():
    wl = workloads.protein(n=2_000, seed=951)
    got, default = _cells_by_kind(wl, 0)
    same, sixty = _cells_by_kind(wl, 60)
    assert sixty == default
    # Whole-warp strips (32 lanes) finish a pair in the fewest steps.
    whole_warp = [sum(_cells_by_kind(wl, s)[1].get(k, 0) for k in (5, 6, 28, 29)) for s in (1, 60, 100_000)]
    assert whole_warp[0] >= whole_warp[1] > whole_warp[2], whole_warp
    for g, w in zip(same, got):
        assert np.array_equal(g, w)
