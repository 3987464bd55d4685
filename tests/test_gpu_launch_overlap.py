"""Launches of long pairs and of the rest of a batch share the GPU: a pair
that keeps one warp busy for tens of milliseconds (the hybrid class, or the
big class without strip teams) holds up neither the other classes nor the
long class.

The device trace (option "trace") gives every launch's first start and last
end; results come from the oracle.
"""
import numpy as np
import pytest

import ipuma_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

PROTEIN = dict(gap_init=-10, gap_extend=-1, similarity="blosum62", datatype="aa")
DNA = dict(gap_init=0, gap_extend=-1, match=5, mismatch=-4, ambiguity=-4)


def _mutated(rng, a, letters, rate):
    b = a.copy()
    at = rng.random(a.size) < rate
    b[at] = rng.choice(letters, int(at.sum()))
    return b


# name: scoring, letters, bits, pairs, |A| of the one-warp pair, of three long
# pairs, team_warps
@pytest.mark.parametrize("sw,letters,bits,n,huge,longer,team_warps", [
    (PROTEIN, range(20), 5, 30_000, 14_000, 4_000, 8),   # hybrid class, the long pairs in a team
    (PROTEIN, range(20), 5, 30_000, 14_000, 4_000, 0),   # hybrid and long class
    (PROTEIN, range(20), 8, 30_000, 7_500, 4_000, 0),    # big and long class
    (DNA, range(1, 5), 2, 150_000, 13_500, 3_000, 0),    # hybrid class beside a launch per class
])
def test_one_long_pair_holds_up_nothing(sw, letters, bits, n, huge, longer, team_warps):
    rng = np.random.default_rng(921)
    letters = np.array(letters, np.uint8)
    few = 300
    a_list = [rng.choice(letters, int(k)) for k in rng.integers(40, 401, few)]
    b_list = [_mutated(rng, a, letters, 0.3) for a in a_list]
    for k in [longer] * 3 + [huge]:
        a_list.append(rng.choice(letters, k))
        b_list.append(_mutated(rng, a_list[-1], letters, 0.005))
    codes, a_off, a_len, b_off, b_len = oracle.pack_pairs(a_list, b_list)
    k = np.concatenate([np.arange(n) % few, np.arange(few, few + 4)])
    pairs = ib.make_pairs(a_off[k], a_len[k], b_off[k], b_len[k])
    sim = oracle.select_matrix(sw.get("similarity", "na"), sw.get("match", 1), sw.get("mismatch", -1),
                               sw.get("ambiguity", -1))
    want = oracle.sw_batch(codes, a_off, a_len, b_off, b_len, sim, sw["gap_init"], sw["gap_extend"],
                           forward_only=True)
    with ib.Engine(ib.sw_config(**sw), ib.algo_config(forward_only=True)) as e:
        e.set_option("autotune", 0)
        e.set_option("team_warps", team_warps)
        e.set_option("trace", 1)
        for _ in range(2):  # the first call loads the kernels
            if bits == 8:
                got = e.compare(codes, pairs)
            else:
                got = e.compare_packed(ib.pack_codes(codes, bits), codes.size, pairs, bits=bits)
        st = e.stats()
    for g, w, name in zip(got, want, ("score", "arange", "brange")):
        assert np.array_equal(g, w[k]), name
    spans = [(st.trace_kind[i], st.trace_start_ms[i], st.trace_end_ms[i]) for i in range(st.n_trace)]
    one_warp = [s for s in spans if s[0] == 20]  # IPUMA_KERNEL_S16_HYBRID: hybrid and big class
    assert len(one_warp) == 1 and len(spans) >= 4, spans
    for kind, start, end in spans:
        if kind != 7:  # the s32 rerun follows every class
            assert start < 0.5 * (one_warp[0][1] + one_warp[0][2]), spans
