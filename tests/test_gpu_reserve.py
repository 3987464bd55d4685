"""ipuma_gpu_reserve: after it, a call of up to the stated pairs and lengths
allocates no device memory -- a smaller call neither, whichever classes, team
sizes and code widths it runs."""
import numpy as np
import pytest
import torch

import ipuma_b200 as ib

pytestmark = pytest.mark.gpu

DNA = dict(gap_init=0, gap_extend=-1)
PROTEIN = dict(gap_init=-10, gap_extend=-1, similarity="blosum62", datatype="aa")


def _call(eng, bits, protein, n, max_a, max_b):
    """n unrelated pairs, one of the longest sequences, through the device call."""
    rng = np.random.default_rng(941)
    lens = np.stack([rng.integers(1, 101, n), rng.integers(1, 101, n)])
    lens[:, 0] = max_a, max_b
    lens = np.minimum(lens, [[max_a], [max_b]])
    codes = rng.integers(0, 20, 200_000) if protein else rng.integers(1, 5, 200_000)
    text = ib.pack_codes(codes.astype(np.uint8), bits) if bits != 8 else codes.astype(np.uint8)
    buf = torch.zeros(text.size + 16, dtype=torch.uint8, device="cuda")
    buf[:text.size] = torch.from_numpy(text).cuda()
    at = rng.integers(0, 200_000 - 10_000, (2, n))
    pairs = torch.from_numpy(ib.make_pairs(at[0], lens[0], at[1], lens[1]).view(np.uint8)).cuda()
    out = torch.zeros(3, n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    args = (pairs.data_ptr(), n, max_a, max_b, out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr())
    if bits == 8:
        eng.compare_device(buf.data_ptr(), codes.size, *args)
    else:
        eng.compare_device_packed(buf.data_ptr(), codes.size, bits, *args)
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("sw,bits,n,max_a,max_b", [
    (DNA, 2, 4_000, 3_000, 1_000),     # teams of six warps, of two for |A| of 1,000
    (DNA, 2, 160_000, 4_000, 500),     # a launch per class; one over all of them below 150,000 pairs
    (PROTEIN, 8, 25_000, 5_000, 5_000)])
def test_smaller_calls_allocate_nothing(sw, bits, n, max_a, max_b):
    protein = sw is PROTEIN
    shapes = [(m, a, b) for m in (n, n // 2, 19_999, 300) if m <= n
              for a in (max_a, 2_600, 2_100, 1_600, 1_000, 513, 512) if a <= max_a for b in (max_b, max_b // 2)]
    # The first call of a kernel loads it: that is not the engine's memory.
    with ib.Engine(ib.sw_config(**sw), ib.algo_config(forward_only=True)) as warm:
        warm.set_option("autotune", 0)
        for m, a, b in shapes:
            _call(warm, bits, protein, m, a, b)
    # A new engine per shape: memory one call took would hide what the next lacks.
    for m, a, b in shapes:
        with ib.Engine(ib.sw_config(**sw), ib.algo_config(forward_only=True)) as e:
            e.set_option("autotune", 0)
            e.reserve(n, max_a, max_b)
            took = _call(e, bits, protein, m, a, b)
            assert took == 0, "%d pairs of %d x %d after a reservation of %d, %d x %d: %d bytes" % (m, a, b, n, max_a,
                                                                                                   max_b, took)
