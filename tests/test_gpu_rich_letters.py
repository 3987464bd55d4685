"""Near-identical proteins of letters that score far above the mean (C, W, H):
their scores pass what the two-tag-bit lanes hold at lengths where an average
protein's do not.  They go to lanes that hold them instead of running twice.

Expected results come from the oracle; every field has to be equal.
"""
import numpy as np
import pytest

import ipuma_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

RICH = np.array([4, 8, 17], np.uint8)  # C, H, W


def _batch(rng, n, share):
    a_list, b_list = [], []
    for _ in range(n):
        a = rng.integers(0, 20, int(rng.integers(700, 1500))).astype(np.uint8)
        rich = rng.random(a.size) < share
        a[rich] = rng.choice(RICH, int(rich.sum()))
        b = a.copy()
        at = rng.random(a.size) < 0.02
        b[at] = rng.integers(0, 20, int(at.sum()))
        k = int(rng.integers(300, 400))  # a gap, so that the main diagonal scores little
        b = np.concatenate([b[:k], b[k + 3:]])
        a_list.append(a)
        b_list.append(b)
    return oracle.pack_pairs(a_list, b_list)


@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("bits", [8, 5])
@pytest.mark.parametrize("n,share", [(60, 0.9), (60, 0.4), (5_000, 0.9)])
def test_rich_pairs_run_once(n, share, bits, forward_only):
    rng = np.random.default_rng(961)
    codes, a_off, a_len, b_off, b_len = _batch(rng, 60, share)
    k = np.arange(n) % 60
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, oracle.select_matrix("blosum62"), -10, -1,
                           forward_only=forward_only)
    assert want[0].max() > 7_839  # what the lanes hold: 8,191 less 32 steps of the largest score
    with ib.Engine(ib.sw_config(-10, -1, similarity="blosum62", datatype="aa"),
                   ib.algo_config(forward_only=forward_only)) as e:
        e.set_option("autotune", 0)
        got = e.compare(codes, pairs) if bits == 8 else e.compare_packed(ib.pack_codes(codes, bits), codes.size, pairs,
                                                                         bits=bits)
        st = e.stats()
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        assert np.array_equal(g, w[k]), name
    assert st.overflow_reruns == 0


@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("bits", [8, 4, 2])
def test_letters_of_unequal_scores_in_dna(bits, forward_only):
    """N scoring above 0 but below a match: the letters decide for DNA too."""
    rng = np.random.default_rng(962)
    a_list = [rng.integers(1, 5, int(k)).astype(np.uint8) for k in rng.integers(300, 1300, 80)]
    b_list = [np.concatenate([a[:100], a[103:]]) for a in a_list]
    if bits != 2:
        for a in a_list[::2]:  # unknown letters
            a[rng.random(a.size) < 0.3] = 0
    codes, a_off, a_len, b_off, b_len = oracle.pack_pairs(a_list, b_list)
    pairs = ib.make_pairs(a_off, a_len, b_off, b_len)
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, oracle.select_matrix("na", 5, -4, 1), 0, -1,
                           forward_only=forward_only)
    with ib.Engine(ib.sw_config(0, -1, 5, -4, 1), ib.algo_config(forward_only=forward_only)) as e:
        e.set_option("autotune", 0)
        got = e.compare(codes, pairs) if bits == 8 else e.compare_packed(ib.pack_codes(codes, bits), codes.size, pairs,
                                                                         bits=bits)
        st = e.stats()
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        assert np.array_equal(g, w), name
    assert st.overflow_reruns == 0
