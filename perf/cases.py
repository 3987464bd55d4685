"""Workloads whose speed this repository tracks: batches of local alignments
through the engine's public calls, from one request of a few pairs to a
million reads.

Sequences are drawn like ``ipuma-lib_b200/python/workloads.py`` draws them
(same length distributions, mutation rates, scorings), on the GPU so that a
million pairs take a moment.  Shapes:

* ``plain``   A = 150 letters, B of U[150, 300] (short reads on windows)
* ``reads``   A of U[50, 250], B lognormal (median 300) in [100, 1000], 10 %
              unrelated pairs
* ``short``   A and B of U[100, 200] (read against read)
* ``protein`` A gamma (mean 350) in [30, 2000], B its mutated copy
* ``tailed``  as protein, 90 % U[50, 400], 9 % U[400, 2000], 1 % U[2000, 8000]
              and 0.5 % near-identical pairs of 7000 to 8000 residues
* ``long``    unrelated A and B of U[0.8 L, L]
"""
from __future__ import annotations

import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ipuma-lib_b200", "python")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ipuma_b200 as ib  # noqa: E402

# Robinson & Robinson (1991) residue frequencies, amino-acid codes 0..19.
AA_FREQ = [0.07805, 0.05129, 0.04487, 0.05364, 0.01925, 0.04264, 0.06295, 0.07377, 0.02199, 0.05142,
           0.09019, 0.05744, 0.02243, 0.03856, 0.05203, 0.07120, 0.05841, 0.01330, 0.03216, 0.06441]
# BLOSUM62 of the amino-acid codes 0..19.
BLOSUM62 = """
 4 -1 -2 -2  0 -1 -1  0 -2 -1 -1 -1 -1 -2 -1  1  0 -3 -2  0
-1  5  0 -2 -3  1  0 -2  0 -3 -2  2 -1 -3 -2 -1 -1 -3 -2 -3
-2  0  6  1 -3  0  0  0  1 -3 -3  0 -2 -3 -2  1  0 -4 -2 -3
-2 -2  1  6 -3  0  2 -1 -1 -3 -4 -1 -3 -3 -1  0 -1 -4 -3 -3
 0 -3 -3 -3  9 -3 -4 -3 -3 -1 -1 -3 -1 -2 -3 -1 -1 -2 -2 -1
-1  1  0  0 -3  5  2 -2  0 -3 -2  1  0 -3 -1  0 -1 -2 -1 -2
-1  0  0  2 -4  2  5 -2  0 -3 -3  1 -2 -3 -1  0 -1 -3 -2 -2
 0 -2  0 -1 -3 -2 -2  6 -2 -4 -4 -2 -3 -3 -2  0 -2 -2 -3 -3
-2  0  1 -1 -3  0  0 -2  8 -3 -3 -1 -2 -1 -2 -1 -2 -2  2 -3
-1 -3 -3 -3 -1 -3 -3 -4 -3  4  2 -3  1  0 -3 -2 -1 -3 -1  3
-1 -2 -3 -4 -1 -2 -3 -4 -3  2  4 -2  2  0 -3 -2 -1 -2 -1  1
-1  2  0 -1 -3  1  1 -2 -1 -3 -2  5 -1 -3 -1  0 -1 -3 -2 -2
-1 -1 -2 -3 -1  0 -2 -3 -2  1  2 -1  5  0 -2 -1 -1 -1 -1  1
-2 -3 -3 -3 -2 -3 -3 -3 -1  0  0 -3  0  6 -4 -2 -2  1  3 -1
-1 -2 -2 -1 -3 -1 -1 -2 -2 -3 -3 -1 -2 -4  7 -1 -1 -4 -3 -2
 1 -1  1  0 -1  0  0  0 -1 -2 -2  0 -1 -2 -1  4  1 -3 -2 -2
 0 -1  0 -1 -1 -1 -1 -2 -2 -1 -1 -1 -1 -2 -1  1  5 -2 -2  0
-3 -3 -4 -4 -2 -2 -3 -2 -2 -3 -2 -3 -1  1 -4 -3 -2 11  2 -3
-2 -2 -2 -3 -2 -1 -2 -3  2 -1 -1 -2 -1  3 -3 -2 -2  2  7 -1
 0 -3 -3 -3 -1 -2 -2 -3 -3  3  1 -2  1 -1 -2 -2  0 -3 -1  4
"""

# Scorings: unit costs (the default driver's), a read mapper's, and BLOSUM62
# with gap open 11 / extend 1 (a gap of length L costs 11 + (L - 1)).
SCORING = {
    "unit": dict(gap_init=0, gap_extend=-1, match=1, mismatch=-1, ambiguity=-1, similarity="na", datatype="na"),
    "mapper": dict(gap_init=-4, gap_extend=-2, match=2, mismatch=-4, ambiguity=-1, similarity="na", datatype="na"),
    "blosum62": dict(gap_init=-10, gap_extend=-1, match=1, mismatch=-1, ambiguity=-1, similarity="blosum62",
                     datatype="aa"),
}

# call: "device" buffers in GPU memory; "host" numpy buffers, pinned ones in
# the large batches; "wire" the batch format of prepare_remote.  bits: width
# of a residue (8 = one byte, else packed).  starts: the reverse pass gives
# start coordinates too.
_CASES = [
    # One request of a service: a handful of reads, latency only.
    dict(name="request_dna_64", call="host", shape="reads", pairs=64, scoring="unit", bits=8, starts=True),
    # A query against a few hundred database proteins, score and end only.
    dict(name="request_protein_500", call="host", shape="protein", pairs=500, scoring="blosum62", bits=8,
         starts=False),
    # A batch of a mapping loop whose buffers stay in place (graph replay).
    dict(name="dna_plain_10k", call="device", shape="plain", pairs=10_000, scoring="unit", bits=2, starts=False,
         graphs=True),
    # A batch of reads with ambiguity letters and a mapper's scoring.
    dict(name="dna_iupac_47k", call="device", shape="reads", pairs=47_001, scoring="mapper", bits=4, starts=False),
    # The default driver's batch: one wire buffer, start coordinates.
    dict(name="dna_wire_100k", call="wire", shape="short", pairs=100_003, scoring="unit", bits=8, starts=True),
    # Reads resident on the GPU, full alignments.
    dict(name="dna_reads_300k_starts", call="device", shape="reads", pairs=300_000, scoring="unit", bits=2,
         starts=True),
    # The benchmark's batch, on resident buffers and from host buffers.
    dict(name="dna_reads_1m", call="device", shape="reads", pairs=1_000_000, scoring="unit", bits=2, starts=False),
    dict(name="dna_reads_1m_host", call="host", shape="reads", pairs=1_000_000, scoring="unit", bits=2,
         starts=False),
    # Protein search: full alignments of a hit list, and a large score pass.
    dict(name="protein_20k_starts", call="device", shape="protein", pairs=20_011, scoring="blosum62", bits=8,
         starts=True),
    dict(name="protein_200k", call="device", shape="protein", pairs=200_000, scoring="blosum62", bits=5,
         starts=False),
    # Lengths with a heavy tail (some scores pass 16 bits).
    dict(name="protein_tailed_60k", call="device", shape="tailed", pairs=60_000, scoring="blosum62", bits=5,
         starts=False),
    # A few long pairs: fewer pairs than the GPU has warps.
    dict(name="protein_long_296", call="device", shape="long", pairs=296, length=6000, scoring="blosum62", bits=8,
         starts=False),
]


def listed():
    return [dict(c) for c in _CASES]


def draw(rng):
    def size(lo, hi):
        return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))

    kind = rng.choice(["request", "dna", "dna", "wire", "protein", "protein", "tailed", "long"])
    starts = rng.random() < 0.4
    if kind == "request":
        shape = rng.choice(["reads", "protein"])
        return dict(call="host", shape=shape, pairs=size(1, 4096), bits=8, starts=starts,
                    scoring="blosum62" if shape == "protein" else "unit")
    if kind == "dna":
        bits = rng.choice([2, 2, 4, 8])
        return dict(call=rng.choice(["device", "device", "host"]), shape=rng.choice(["plain", "reads", "short"]),
                    pairs=size(4096, 400_000), scoring="mapper" if bits == 4 else "unit", bits=bits, starts=starts)
    if kind == "wire":
        return dict(call="wire", shape="short", pairs=size(500, 150_000), scoring="unit", bits=8, starts=starts)
    if kind == "long":
        length = size(1500, 8000)
        return dict(call="device", shape="long", pairs=max(1, int(size(16, 1200) * min(1.0, (3000 / length) ** 2))),
                    length=length, scoring="blosum62", bits=rng.choice([5, 8]), starts=starts)
    return dict(call="device", shape=kind, pairs=size(1000, 100_000 if kind == "protein" else 30_000),
                scoring="blosum62", bits=rng.choice([5, 8]), starts=starts)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _lengths(case, seed):
    """(|A|, target |B|, unrelated, near-identical) per pair."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, shape = case["pairs"], case["shape"]
    none = np.zeros(n, bool)
    if shape == "plain":
        return np.full(n, 150, np.int64), rng.integers(150, 301, n), none, none
    if shape == "reads":
        a = rng.integers(50, 251, n)
        b = np.clip(np.round(np.exp(rng.normal(np.log(300.0), 0.5, n))), 100, 1000).astype(np.int64)
        return a, b, rng.random(n) < 0.10, none
    if shape == "short":
        return rng.integers(100, 201, n), rng.integers(100, 201, n), rng.random(n) < 0.10, none
    if shape == "long":
        lo = max(1, int(0.8 * case["length"]))
        return (rng.integers(lo, case["length"] + 1, n), rng.integers(lo, case["length"] + 1, n), np.ones(n, bool),
                none)
    if shape == "protein":
        a = np.clip(np.round(rng.gamma(2.0, 175.0, n)), 30, 2000).astype(np.int64)
        return a, a, none, none
    u = rng.random(n)
    a = np.where(u < 0.90, rng.integers(50, 401, n),
                 np.where(u < 0.99, rng.integers(400, 2001, n), rng.integers(2000, 8001, n)))
    ident = np.zeros(n, bool)
    ident[rng.choice(n, int(round(0.005 * n)), replace=False)] = True
    a = np.where(ident, rng.integers(7000, 8001, n), a).astype(np.int64)
    return a, a, none, ident


def _matrix62(dev):
    return torch.tensor([int(x) for x in BLOSUM62.split()], device=dev).reshape(20, 20)


def _sequences(case, seed, dev="cuda"):
    """(codes uint8, a_off, a_len, b_off, b_len) on the GPU: every A, then
    every B."""
    a_np, t_np, unrel_np, ident_np = _lengths(case, seed)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    n = case["pairs"]
    protein = case["scoring"] == "blosum62"
    a_len, target = torch.from_numpy(a_np).to(dev), torch.from_numpy(t_np.astype(np.int64)).to(dev)
    unrel, ident = torch.from_numpy(unrel_np).to(dev), torch.from_numpy(ident_np).to(dev)
    edges = torch.tensor(AA_FREQ, device=dev).cumsum(0)
    edges = (edges / edges[-1])[:19].contiguous()

    def rand(m):
        return torch.rand(m, generator=g, device=dev)

    def letters(m):
        if protein:
            return torch.bucketize(rand(m), edges, right=True).to(torch.uint8)
        return torch.randint(1, 5, (m,), generator=g, device=dev, dtype=torch.uint8)

    def per_pair(lo, hi):
        return lo + (hi - lo) * rand(n)

    total = int(a_np.sum())
    a_all = letters(total)
    pair = torch.repeat_interleave(torch.arange(n, device=dev), a_len)
    if protein:
        sub_rate = torch.where(ident, per_pair(0.0, 0.01), per_pair(0.20, 0.60))
        indel_rate = torch.where(ident, torch.zeros(n, device=dev), per_pair(0.01, 0.05))
        max_indel = 5
    elif case["shape"] == "plain":
        sub_rate, indel_rate, max_indel = per_pair(0.05, 0.05), per_pair(0.02, 0.02), 1
    else:
        sub_rate, indel_rate, max_indel = per_pair(0.03, 0.15), per_pair(0.01, 0.05), 3

    # substitutions
    core = a_all.clone()
    at = torch.nonzero(rand(total) < sub_rate[pair]).flatten()
    if protein:
        p = torch.tensor(AA_FREQ, device=dev)
        w = p[None, :] * torch.pow(2.0, _matrix62(dev).float() / 2.0)
        w.fill_diagonal_(0.0)
        cdf = (w / w.sum(1, keepdim=True)).cumsum(1)
        for x in range(20):
            here = at[a_all[at] == x]
            core[here] = torch.bucketize(rand(here.numel()), cdf[x].contiguous(), right=True).clamp_(max=19).to(
                torch.uint8)
    else:
        shift = torch.randint(1, 4, (at.numel(),), generator=g, device=dev, dtype=torch.uint8)
        core[at] = (a_all[at] - 1 + shift) % 4 + 1
    # indel events, half deletions and half insertions
    ev = torch.nonzero(rand(total) < indel_rate[pair]).flatten()
    ln = torch.randint(1, max_indel + 1, (ev.numel(),), generator=g, device=dev)
    is_del = rand(ev.numel()) < 0.5
    pair_end = a_len.cumsum(0)
    dpos, dlen = ev[is_del], ln[is_del]
    diff = torch.zeros(total + 1, dtype=torch.int32, device=dev)
    one = torch.ones(dpos.numel(), dtype=torch.int32, device=dev)
    diff.index_add_(0, dpos, one)
    diff.index_add_(0, torch.minimum(dpos + dlen, pair_end[pair[dpos]]), -one)
    count = (diff[:-1].cumsum(0) <= 0).long()
    count[ev[~is_del]] += ln[~is_del]
    src = torch.repeat_interleave(torch.arange(total, device=dev), count)
    kept = torch.ones(src.numel(), dtype=torch.bool, device=dev)
    kept[1:] = src[1:] != src[:-1]
    core = torch.where(kept, core[src], letters(src.numel()))
    core_pair = pair[src]
    core_len = torch.bincount(core_pair, minlength=n)
    del src, kept, count, diff, ev, ln, is_del

    # B: the mutated copy inside random flanks, or random letters
    if protein and case["shape"] != "long":
        target = core_len.clamp(min=1)
    b_len = torch.where(unrel, target, torch.maximum(target, core_len))
    b_start = b_len.cumsum(0) - b_len
    b_all = letters(int(b_len.sum()))
    slack = (b_len - core_len).clamp(min=0)
    left = torch.minimum((rand(n) * (slack + 1)).long(), slack)
    keep = ~unrel[core_pair]
    core_start = core_len.cumsum(0) - core_len
    pos = torch.arange(core.numel(), device=dev) - core_start[core_pair] + (b_start + left)[core_pair]
    b_all[pos[keep]] = core[keep]
    codes = torch.cat([a_all, b_all])
    if case["bits"] == 4:  # about 1 % N and a few other ambiguity letters
        u = rand(codes.numel())
        codes = torch.where(u < 0.01, torch.zeros_like(codes), codes)
        codes = torch.where(u > 0.998, torch.randint(6, 16, (codes.numel(),), generator=g, device=dev,
                                                     dtype=torch.uint8), codes)
    return codes, a_len.cumsum(0) - a_len, a_len, total + b_start, b_len


def _pack(codes, bits):
    """Packed codes with the readable words the device calls ask for."""
    if bits == 8:
        return torch.cat([codes, codes.new_zeros(16)])
    m = codes.numel()
    room = ib.device_packed_bytes(m, bits)
    x = codes - 1 if bits == 2 else codes
    x = torch.cat([x, x.new_zeros(-m % 8)]).reshape(-1, 8).long()
    word = torch.zeros(x.shape[0], dtype=torch.int64, device=codes.device)
    for q in range(8):
        word |= x[:, q] << (bits * q)
    out = torch.stack([(word >> (8 * k)) & 255 for k in range(bits)], 1).to(torch.uint8).flatten()
    return torch.cat([out, out.new_zeros(max(0, room - out.numel()) + 16)])


def _pairs(a_off, a_len, b_off, b_len):
    return ib.make_pairs(a_off.cpu().numpy(), a_len.cpu().numpy(), b_off.cpu().numpy(), b_len.cpu().numpy())


_WIRE_SLOTS = 100  # comparisons per tile of the wire buffer


def _wire_layout(a_len, b_len):
    """Tile byte offsets of each pair's A, and the tile size."""
    n = a_len.numel()
    tile = torch.arange(n, device=a_len.device) // _WIRE_SLOTS
    need = a_len + b_len
    start = need.cumsum(0) - need
    off = start - start[tile * _WIRE_SLOTS]
    return tile, off, int((off + need).max())


def prepare(case, seed):
    codes, a_off, a_len, b_off, b_len = _sequences(case, seed)
    n = case["pairs"]
    sw = ib.sw_config(**SCORING[case["scoring"]])
    st = {"case": case, "n": n, "n_codes": codes.numel()}
    if case["call"] == "wire":
        tile, off, bufsize = _wire_layout(a_len, b_len)
        tiles = (n + _WIRE_SLOTS - 1) // _WIRE_SLOTS
        words = (bufsize + 3) // 4
        seq = torch.zeros(tiles * words * 4, dtype=torch.uint8, device=codes.device)
        for src, ln, at in ((a_off, a_len, off), (b_off, b_len, off + a_len)):
            step = torch.arange(int(ln.sum()), device=codes.device) - torch.repeat_interleave(ln.cumsum(0) - ln, ln)
            seq[torch.repeat_interleave(tile * words * 4 + at, ln) + step] = codes[
                torch.repeat_interleave(src, ln) + step]
        meta = torch.zeros(tiles * _WIRE_SLOTS, 4, dtype=torch.int32, device=codes.device)
        meta[:n] = torch.stack([a_len, off, b_len, off + a_len], 1).to(torch.int32)
        st["inputs"] = np.concatenate([seq.cpu().numpy().view(np.int32), meta.flatten().cpu().numpy()])
        algo = ib.algo_config(tiles_used=tiles, max_ab=200, max_batches=_WIRE_SLOTS, bufsize=bufsize,
                              forward_only=not case["starts"])
        st["engine"] = ib.Engine(sw, algo)
        st["engine"].autotune()
        return st
    eng = st["engine"] = ib.Engine(sw, ib.algo_config(forward_only=not case["starts"]))
    eng.autotune()
    pairs = _pairs(a_off, a_len, b_off, b_len)
    packed = _pack(codes, case["bits"])
    if case["call"] == "host":
        used = ib.packed_bytes(codes.numel(), case["bits"]) if case["bits"] != 8 else codes.numel()
        pinned = n >= 100_000
        out = torch.zeros(3, n, dtype=torch.int32, pin_memory=pinned)
        text = torch.empty(used, dtype=torch.uint8, pin_memory=pinned)
        text.copy_(packed[:used])
        desc = torch.empty(n * 24, dtype=torch.uint8, pin_memory=pinned)
        desc.copy_(torch.from_numpy(pairs.view(np.uint8)))
        st.update(out=out, text=text, desc=desc, codes=text.numpy(), pairs=desc.numpy().view(ib.PAIR_DTYPE),
                  score=out[0].numpy(), arange=out[1].numpy(), brange=out[2].numpy())
        return st
    max_a, max_b = int(a_len.max()), int(b_len.max())
    if case.get("graphs"):
        eng.set_option("graphs", 1)
    eng.reserve(n, max_a, max_b)
    st.update(codes=packed, pairs=torch.from_numpy(pairs.view(np.uint8)).cuda(), max_a=max_a, max_b=max_b,
              out=torch.zeros(3, n, dtype=torch.int32, device="cuda"),
              stream=torch.cuda.current_stream().cuda_stream)
    return st


def run(st):
    case, eng = st["case"], st["engine"]
    if case["call"] == "wire":
        return eng.run_buffer(st["inputs"])
    if case["call"] == "host":
        if case["bits"] == 8:
            eng.compare_into(st["codes"], st["pairs"], st["score"], st["arange"], st["brange"])
        else:
            eng.compare_packed_into(st["codes"], st["n_codes"], st["pairs"], st["score"], st["arange"], st["brange"],
                                    bits=case["bits"])
        return st["score"], st["arange"], st["brange"]
    score, arange, brange = st["out"][0], st["out"][1], st["out"][2]
    args = (st["pairs"].data_ptr(), st["n"], st["max_a"], st["max_b"], score.data_ptr(), arange.data_ptr(),
            brange.data_ptr(), st["stream"])
    if case["bits"] == 8:
        eng.compare_device(st["codes"].data_ptr(), st["n_codes"], *args)
    else:
        eng.compare_device_packed(st["codes"].data_ptr(), st["n_codes"], case["bits"], *args)
    return score, arange, brange


def work(case):
    """Each residue, descriptor and result once; per cell the seven integer
    operations of the recurrence (an alignment has no floating-point work).
    With start coordinates the reverse pass revisits a part of the cells
    that depends on the sequences; the forward pass alone is counted."""
    a, t, _, _ = _lengths(case, 0)
    cells = float(np.dot(a.astype(np.float64), np.maximum(t, a if case["shape"] != "long" else t)))
    residues = float(a.sum() + np.maximum(t, a).sum())
    return {"bytes": residues * case["bits"] / 8 + case["pairs"] * (24 + 12), "flops": 7.0 * cells}


# --------------------------------------------------------------------------
# the answer in plain 64-bit arithmetic
# --------------------------------------------------------------------------
def _similarity(scoring, dev):
    s = SCORING[scoring]
    if s["similarity"] == "blosum62":
        return _matrix62(dev)
    m = torch.full((16, 16), s["mismatch"], dtype=torch.int64, device=dev)  # bases only (codes 1 to 4)
    return m.fill_diagonal_(s["match"])


def _pass(codes, sim, gi, ge, a0, al, da, b0, bl, db):
    """First strict maximum in (row, column) order of one pass per pair:
    (score, column, row)."""
    n, cols, rows = al.numel(), int(al.max()), int(bl.max())
    dev = codes.device
    j = torch.arange(cols, device=dev)
    valid = j[None, :] < al[:, None]
    last = codes.numel() - 1
    acode = codes[(a0[:, None] + da * j[None, :]).clamp_(0, last)].long() * sim.shape[1]
    h = torch.zeros(n, cols, dtype=torch.int64, device=dev)
    f = torch.zeros_like(h)
    shift = -ge * j  # E in the frame where an extension costs nothing
    back = gi + ge * j[None, 1:]
    order = cols - 1 - j
    best = torch.zeros(n, dtype=torch.int64, device=dev)
    bi, bj = torch.zeros_like(best), torch.zeros_like(best)
    flat = sim.flatten()
    for i in range(rows):
        bc = codes[(b0 + db * i).clamp(0, last)].long()
        f = torch.maximum(f + ge, h + (gi + ge))
        s = flat[acode + bc[:, None]]
        s[:, 1:] += h[:, :-1]
        h = torch.maximum(s, f).clamp_(min=0)
        e = torch.cummax(h + shift, 1).values
        h[:, 1:] = torch.maximum(h[:, 1:], e[:, :-1] + back)
        key = torch.where(valid, h * cols + order, -1).amax(1)
        sc = torch.div(key, cols, rounding_mode="floor")
        up = (sc > best) & (i < bl)
        best = torch.where(up, sc, best)
        bi = torch.where(up, i, bi)
        bj = torch.where(up, cols - 1 - key % cols, bj)
    return best, bj, bi


def exact(case, seed):
    # The largest batches would take too long; the ambiguity letters of the
    # 4-bit batches need the whole IUPAC table.
    if case["shape"] == "tailed" or case["bits"] == 4 or case["pairs"] > 400_000 or (
            case["shape"] == "protein" and case["pairs"] > 50_000):
        return None
    codes, a_off, a_len, b_off, b_len = _sequences(case, seed)
    dev, n = codes.device, case["pairs"]
    s = SCORING[case["scoring"]]
    sim, gi, ge = _similarity(case["scoring"], dev), s["gap_init"], s["gap_extend"]
    out = torch.zeros(3, n, dtype=torch.int64, device=dev)
    order = torch.argsort(b_len)
    at = 0
    while at < n:
        m = max(1, min(n - at, 20_000_000 // int(a_len.max())))
        p = order[at:at + m]
        at += m
        sc, ae, be = _pass(codes, sim, gi, ge, a_off[p], a_len[p], 1, b_off[p], b_len[p], 1)
        a_st, b_st = torch.zeros_like(ae), torch.zeros_like(be)
        if case["starts"]:
            on = sc > 0
            _, aj, bj = _pass(codes, sim, gi, ge, a_off[p] + ae, torch.where(on, ae + 1, 1), -1, b_off[p] + be,
                              torch.where(on, be + 1, 1), -1)
            a_st, b_st = torch.where(on, ae - aj, 0), torch.where(on, be - bj, 0)
        out[0, p] = sc
        out[1, p] = a_st | (ae << 16)
        out[2, p] = b_st | (be << 16)
    if case["call"] == "wire":
        slots = (n + _WIRE_SLOTS - 1) // _WIRE_SLOTS * _WIRE_SLOTS
        full = torch.zeros(3, slots, dtype=torch.int64, device=dev)
        full[:, :n] = out
        return full.flatten().cpu().numpy()
    if case["call"] == "host":
        return tuple(x.cpu().numpy() for x in out)
    return out[0], out[1], out[2]
