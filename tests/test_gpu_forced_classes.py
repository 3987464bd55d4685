"""Option tile_k takes every class it lists for every scoring, code width and
batch size.  Scorings whose scaled values pass a byte, and large 2-bit
batches with linear gaps, have kernels for part of the widths only: there
the pairs run in the narrowest strips at least as wide.

Expected results come from the oracle; every field has to be equal.
"""
import numpy as np
import pytest

import ipuma_b200 as ib
import oracle

pytestmark = pytest.mark.gpu


def _batch(rng, n):
    """|A| beside multiples of 64 columns and several strips of them."""
    edges = np.array([1, 63, 64, 65, 80, 95, 96, 97, 112, 127, 128, 129, 192, 193, 255, 256, 257, 385, 513])
    a_list, b_list = [], []
    for k in range(n):
        a = rng.integers(1, 5, edges[k % edges.size]).astype(np.uint8)
        b = rng.integers(1, 5, int(rng.integers(1, 200))).astype(np.uint8)
        if k % 2:
            at = int(rng.integers(0, b.size))
            m = min(a.size, b.size - at)
            b[at:at + m] = a[:m]
            b[at:at + m:19] = 2
        a_list.append(a)
        b_list.append(b)
    return oracle.pack_pairs(a_list, b_list)


def _check(scoring, bits, n, tile_k, forward_only):
    gi, ge, match, mismatch = scoring
    codes, a_off, a_len, b_off, b_len = _batch(np.random.default_rng(931), min(n, 190))
    k = np.arange(n) % a_len.size
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, oracle.select_matrix("na", match, mismatch, mismatch),
                           gi, ge, forward_only=forward_only)
    with ib.Engine(ib.sw_config(gi, ge, match, mismatch, mismatch), ib.algo_config(forward_only=forward_only)) as e:
        e.set_option("autotune", 0)
        e.set_option("tile_k", tile_k)
        got = e.compare(codes, pairs) if bits == 8 else e.compare_packed(ib.pack_codes(codes, bits), codes.size, pairs,
                                                                         bits=bits)
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        bad = np.nonzero(g != w[k])[0]
        assert bad.size == 0, "tile_k %d %s: %d differ, first %d" % (tile_k, name, bad.size, bad[0])


@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("bits", [8, 2])
@pytest.mark.parametrize("tile_k", [1, 2, 3, 4, 5, 6] + list(range(8, 22)))
def test_unscaled_scores(tile_k, bits, forward_only):
    _check((-7, -3, 50, -40), bits, 190, tile_k, forward_only)


@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("n", [149_999, 150_000])
@pytest.mark.parametrize("tile_k", [17, 18, 19, 20, 21])
def test_eight_lane_classes_at_both_sides_of_the_large_batches(tile_k, n, forward_only):
    _check((0, -1, 1, -1), 2, n, tile_k, forward_only)
