"""The 16-bit lanes of the wavefront classes (tag_pass): every strip width at
its edges, the lanes each scoring picks (linear gaps, affine, any score),
and scores around the limits their tag bits leave.

Expected results come from the oracle; every field has to be equal.
"""
import numpy as np
import pytest

import ipuma_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

# gap_init, gap_extend, match, mismatch: linear gaps; affine; linear gaps
# whose scaled values pass a byte (affine lanes); any score (unscaled lanes).
SCORINGS = {"linear": (0, -1, 1, -1), "affine": (-4, -2, 2, -4), "linear_wide": (0, -3, 6, -5),
            "any": (-7, -3, 50, -40)}


def _pairs_at_edges(rng, n):
    """n pairs whose |A| sits on and beside multiples of 16 columns up to
    three strips of 512, |B| short and long; half of them related."""
    edges = np.array([1, 2, 15, 16, 17] + [16 * k + d for k in range(4, 17) for d in (-1, 0, 1)] +
                     [383, 384, 385, 511, 512, 513, 1023, 1024, 1025, 1536])
    a_len = edges[np.arange(n) % edges.size]
    a_list, b_list = [], []
    for la in a_len:
        a = rng.integers(1, 5, la).astype(np.uint8)
        lb = int(rng.integers(1, 90))
        if rng.random() < 0.5:
            k = int(rng.integers(0, la))
            b = np.concatenate([rng.integers(1, 5, int(rng.integers(0, 6))).astype(np.uint8), a[k:k + lb]])
        else:
            b = rng.integers(1, 5, lb).astype(np.uint8)
        a_list.append(a)
        b_list.append(b)
    return oracle.pack_pairs(a_list, b_list)


def _run(scoring, forward_only, codes, pairs, bits, **opts):
    gi, ge, match, mismatch = SCORINGS[scoring]
    with ib.Engine(ib.sw_config(gi, ge, match, mismatch, mismatch), ib.algo_config(forward_only=forward_only)) as e:
        for k, v in opts.items():
            e.set_option(k, v)
        got = e.compare(codes, pairs) if bits == 8 else e.compare_packed(ib.pack_codes(codes, bits), codes.size,
                                                                         pairs, bits=bits)
        return got, e.stats()


def _same(got, want, label):
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        bad = np.nonzero(g != w)[0]
        assert bad.size == 0, "%s %s: %d differ, first %d: %d vs %d" % (label, name, bad.size, bad[0], g[bad[0]],
                                                                        w[bad[0]])


@pytest.mark.parametrize("scoring", list(SCORINGS))
@pytest.mark.parametrize("bits,n", [(8, 300), (2, 300), (2, 49_000)])
def test_strip_edges(scoring, bits, n):
    """Small batches use 16-lane groups, large ones with 2-bit codes and
    linear gaps 8-lane groups."""
    rng = np.random.default_rng(901)
    codes, a_off, a_len, b_off, b_len = _pairs_at_edges(rng, 300)
    k = np.arange(n) % 300
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    gi, ge, match, mismatch = SCORINGS[scoring]
    sim = oracle.select_matrix("na", match, mismatch, mismatch)
    for fwd in (True, False):
        want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, sim, gi, ge, forward_only=fwd)
        got, _ = _run(scoring, fwd, codes, pairs, bits)
        _same(got, [w[k] for w in want], "%s bits %d n %d fwd %s" % (scoring, bits, n, fwd))


@pytest.mark.parametrize("scoring,tile_k,lengths", [
    ("linear", 4, (2000, 2014, 2015, 2016, 2047, 2048, 2100)),    # 4 tag bits: 2,047 points
    ("linear", 0, (2014, 2015, 2016, 2017, 2048, 2400)),          # widest strips or the long class
    ("affine", 6, (4000, 4063, 4064, 4095, 4096, 4200)),          # 2 tag bits: 8,191 points
    ("affine", 0, (4063, 4064, 4065, 4096))])
def test_scores_around_the_tag_limit(scoring, tile_k, lengths):
    """Identical pairs whose scores lie around what the lanes hold: past it
    the pair is rerun in 32 bits (or was given to the long class)."""
    rng = np.random.default_rng(902)
    a_list = [rng.integers(1, 5, la).astype(np.uint8) for la in lengths]
    codes, a_off, a_len, b_off, b_len = oracle.pack_pairs(a_list, a_list)
    pairs = ib.make_pairs(a_off, a_len, b_off, b_len)
    gi, ge, match, mismatch = SCORINGS[scoring]
    sim = oracle.select_matrix("na", match, mismatch, mismatch)
    for fwd in (True, False):
        want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, sim, gi, ge, forward_only=fwd)
        got, st = _run(scoring, fwd, codes, pairs, 8, tile_k=tile_k)
        _same(got, want, "%s tile_k %d fwd %s" % (scoring, tile_k, fwd))
        if tile_k:
            assert st.overflow_reruns >= 1


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1025, 4095, 4096, 4097])
def test_list_of_a_small_batch(n):
    """The one-block pre-pass (up to 4,096 pairs) and the histogram one:
    every pair gets its own result, empty pairs zero, whatever their order."""
    rng = np.random.default_rng(903)
    codes, a_off, a_len, b_off, b_len = _pairs_at_edges(rng, 120)
    k = rng.integers(0, 120, n)
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    empty = rng.random(n) < 0.05
    pairs["b_len"][empty] = 0
    gi, ge, match, mismatch = SCORINGS["affine"]
    sim = oracle.select_matrix("na", match, mismatch, mismatch)
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, sim, gi, ge, forward_only=False)
    got, _ = _run("affine", False, codes, pairs, 8)
    _same(got, [np.where(empty, 0, w[k]) for w in want], "n %d" % n)


@pytest.mark.parametrize("n,team_warps", [(3, 8), (40, 8), (40, 6), (40, 0)])
def test_high_scores_in_teams(n, team_warps):
    """Near-identical proteins scoring above int16: strip teams of biased
    halves (one, two or four teams a block), or one warp each."""
    rng = np.random.default_rng(904)
    a_list = [rng.integers(0, 20, int(la)).astype(np.uint8) for la in rng.integers(6600, 7400, n)]
    b_list = []
    for a in a_list:
        b = a.copy()
        at = rng.integers(0, a.size, 20)
        b[at] = rng.integers(0, 20, 20)
        b_list.append(b)
    codes, a_off, a_len, b_off, b_len = oracle.pack_pairs(a_list, b_list)
    pairs = ib.make_pairs(a_off, a_len, b_off, b_len)
    for fwd in (True, False):
        with ib.Engine(ib.sw_config(-10, -1, similarity="blosum62", datatype="aa"),
                       ib.algo_config(forward_only=fwd)) as e:
            e.set_option("team_warps", team_warps)
            got = e.compare(codes, pairs)
            st = e.stats()
        want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, oracle.select_matrix("blosum62"), -10, -1,
                               forward_only=fwd)
        assert want[0].min() > 32767
        _same(got, want, "n %d warps %d fwd %s" % (n, team_warps, fwd))
        assert st.overflow_reruns == 0 and st.s32_pairs == n
