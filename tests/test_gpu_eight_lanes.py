"""8-lane groups of the 2-bit linear-gap classes (batches of 150,000 pairs
and more): strips of every width they have, forced and chosen by cost, with
and without start coordinates, |A| on both sides of one and several strips.

Expected results come from the oracle; every field has to be equal.
"""
import numpy as np
import pytest

import ipuma_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

N = 150_000     # smallest batch that runs them
DISTINCT = 320  # distinct pairs, repeated N / DISTINCT times


def _batch(rng):
    """Pairs with |A| beside multiples of 16 columns from 64 to 256 (the strip
    widths), twice and three times those; |B| of 1 to 300; half related."""
    edges = np.array([1, 7, 8, 63, 64, 65] + [m * 16 * k + d for m in (1, 2, 3) for k in range(4, 17)
                                              for d in (-1, 0, 1)])
    a_len = edges[np.arange(DISTINCT) % edges.size]
    a_list, b_list = [], []
    for la in a_len:
        a = rng.integers(1, 5, la).astype(np.uint8)
        b = rng.integers(1, 5, int(rng.integers(1, 301))).astype(np.uint8)
        if rng.random() < 0.5:
            k, at = int(rng.integers(0, la)), int(rng.integers(0, b.size))
            m = min(la - k, b.size - at)
            b[at:at + m] = a[k:k + m]
            b[at:at + m:17] = 1
        a_list.append(a)
        b_list.append(b)
    return oracle.pack_pairs(a_list, b_list)


# 0: by cost; 1, 2, 3, 4: 64, 128, 192, 256 columns; 8 .. 16: 96, 160, 224,
# 80, 112, 144, 176, 208, 240; 5, 6: whole-warp strips of 384 and 512.
@pytest.mark.parametrize("forward_only", [True, False])
@pytest.mark.parametrize("tile_k", [0, 1, 2, 3, 4, 5, 6, 8, 9, 10, 11, 12, 13, 14, 15, 16])
def test_every_strip_width(tile_k, forward_only):
    rng = np.random.default_rng(911)
    codes, a_off, a_len, b_off, b_len = _batch(rng)
    k = np.arange(N) % DISTINCT
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, oracle.select_matrix("na", 1, -1, -1), 0, -1,
                           forward_only=forward_only)
    with ib.Engine(ib.sw_config(0, -1, 1, -1, -1), ib.algo_config(forward_only=forward_only)) as e:
        e.set_option("tile_k", tile_k)
        got = e.compare_packed(ib.pack_codes(codes, 2), codes.size, pairs, bits=2)
        st = e.stats()
    if tile_k == 0:
        assert st.launches >= 15  # a launch per class, not one over all of them
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        bad = np.nonzero(g != w[k])[0]
        assert bad.size == 0, "tile_k %d %s: %d differ, first %d: %d vs %d" % (tile_k, name, bad.size, bad[0],
                                                                             g[bad[0]], w[k][bad[0]])
