"""What the speed of this framework is measured on: batches of sequence pairs
through its public calls (``Aligner.align_arrays`` on host buffers,
``Aligner.align_device`` on CUDA tensors), from one pair to long noisy reads.

Sizes follow the repository's own workloads (tsunami_pact_b200/datasets.py):
c1 (150 bp), c2 (1 kbp), c3 (10 kbp at 15 %), c4 (uneven, 100 bp - 20 kbp) and
the long class of c5 (10 - 50 kbp), with fewer pairs where a whole workload
takes seconds.  Pairs are i.i.d. ACGT with equal substitutions, insertions and
deletions, as its generator makes them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tsunami_pact_b200 as T

GB = 1 << 30
# penalty models: constructor arguments, cost of a substitution and of a
# one-base gap, smallest gap extension, unit (gcd of the penalties)
MODELS = {
    "affine": (dict(mismatch=4, gap_opening=6, gap_extension=2), 4, 8, 2, 2),
    "dual": (dict(mismatch=4, gap_opening=6, gap_extension=2, gap_opening2=24, gap_extension2=1), 4, 8, 1, 1),
    "edit": (dict(metric="edit"), 1, 1, 1, 1),
    "indel": (dict(metric="indel"), 2, 1, 1, 1),
    "linear": (dict(mismatch=4, gap_opening=0, gap_extension=2, metric="gap_linear"), 4, 2, 2, 2),
}


def _case(name, via, model, pairs, length, max_length, rate, max_rate, cigar=True, free=0, option=""):
    c = {} if name is None else {"name": name}
    return dict(c, via=via, model=model, pairs=pairs, length=length, max_length=max_length, rate=rate,
                max_rate=max_rate, cigar=cigar, free=free, option=option)


def listed():
    return [
        # one read against one candidate region: a mapper's smallest call
        _case("one_pair_1k", "host", "affine", 1, 1000, 1000, 0.05, 0.05),
        # short-read verification in a mapper's batch (c1)
        _case("reads_150", "host", "affine", 10_000, 150, 150, 0.02, 0.02),
        # accurate 1 kbp reads at scale, data resident on the GPU (c2's shape)
        _case("reads_1k", "device", "affine", 200_000, 1000, 1000, 0.05, 0.05),
        # the same scored only, as in filtering (the reference kernel's own work)
        _case("scores_1k", "device", "affine", 200_000, 1000, 1000, 0.05, 0.05, cigar=False),
        # read overlaps of a few kbp, uneven lengths (the middle class of c5)
        _case("reads_1k_5k", "device", "affine", 5_000, 1000, 5000, 0.05, 0.10),
        # long noisy reads (c3)
        _case("long_10k", "device", "affine", 1_000, 10_000, 10_000, 0.15, 0.15),
        # a mixed run from host memory and back (c4)
        _case("uneven", "host", "affine", 8_000, 100, 20_000, 0.01, 0.15),
        # edit distance with its alignments: clustering, barcodes, contigs
        _case("edit_1k", "device", "edit", 200_000, 1000, 1000, 0.05, 0.05),
        # a read placed in a somewhat longer region: free ends
        _case("semiglobal_1k", "device", "affine", 20_000, 1000, 1000, 0.05, 0.05, free=100),
        # two-piece gaps, the usual model for long indels
        _case("dual_1k", "device", "dual", 20_000, 1000, 1000, 0.05, 0.05),
        # long noisy reads in linear memory
        _case("bidir_10k", "device", "affine", 500, 10_000, 10_000, 0.15, 0.15, option="bidirectional"),
        # very long noisy reads in little memory (the long class of c5)
        _case("lowmem_10k_50k", "device", "affine", 24, 10_000, 50_000, 0.10, 0.20, option="low_memory"),
    ]


def _score(case, length, rate):
    """Expected score of a pair in units of the penalties' gcd."""
    _, x, g1, _, unit = MODELS[case["model"]]
    return length * rate * (x + 2 * g1) / 3.0 / unit


def _cells(case):
    """Expected wavefront cells of a batch: about s^2 / e per pair (s the
    score, both in units), at most (2 s / e) x s; lengths are log-uniform,
    rates uniform."""
    _, _, _, e, unit = MODELS[case["model"]]
    a, b = math.log(case["length"]), math.log(case["max_length"])
    total = 0.0
    for i in range(16):
        L = math.exp(a + (b - a) * (i + 0.5) / 16)
        r = case["rate"] + (case["max_rate"] - case["rate"]) * ((i * 7 % 16) + 0.5) / 16
        s = _score(case, L, r)
        total += min(s, 2 * L * e / unit) * s / (e / unit) + (2 * case["free"] + 3) * s + 1
    return case["pairs"] * total / 16


# Cells a drawn batch may have (half of what the most expensive listed cases
# have per model and option) and bases it may hold.
CELL_CAP = {"affine": 5e9, "dual": 1e9, "edit": 2e9, "indel": 2e9, "linear": 2e9}


def draw(rng):
    def spread(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["plain", "plain", "plain", "scores", "model", "model", "free", "bidirectional", "low_memory"])
    model, cigar, free, option = "affine", True, 0, ""
    lo, hi = 60, 20_000
    if kind == "scores":
        cigar = False
    elif kind == "model":
        model = rng.choice(["dual", "edit", "indel", "linear"])
        cigar = rng.random() < 0.7
        hi = 5_000
    elif kind == "free":
        model = rng.choice(["affine", "edit"])
        hi = 3_000
    elif kind == "bidirectional":
        option, lo = kind, 1_000
    elif kind == "low_memory":
        option, lo, hi = kind, 2_000, 40_000
    length = int(spread(lo, hi))
    max_length = length if rng.random() < 0.5 else min(hi, int(length * spread(1.1, 8)))
    rate = spread(0.01, 0.15)
    max_rate = min(0.2, rate * rng.choice([1.0, 1.0, 1.5, 3.0]))
    if kind == "free":
        free = max(1, int(length * spread(0.02, 0.2)))
    c = _case(None, rng.choice(["host", "device", "device"]), model, 1, length, max_length, rate, max_rate, cigar, free,
              option)
    cap = CELL_CAP[model] / (4 if option == "low_memory" else 2 if option or free else 1)
    most = min(200_000, cap / _cells(c), 1.5e8 / max_length)
    c["pairs"] = max(1, int(spread(1, max(1.0, most))))
    return c


def _lengths(case, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    n = case["pairs"]
    L = np.exp(r.uniform(math.log(case["length"]), math.log(case["max_length"]), n))
    L = np.clip(np.rint(L), case["length"], case["max_length"]).astype(np.int32)
    return L, r.uniform(case["rate"], case["max_rate"], n)


def _batch(case, seed):
    lengths, rates = _lengths(case, seed)
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(seed * 2654435761 % (1 << 62) + 1, lengths, rates)
    if case["free"]:
        # the text is a region around the read's place, the read overhangs a
        # little: unrelated bases at both ends of the text and of the pattern
        r = np.random.Generator(np.random.PCG64(seed + 7))
        f, g = case["free"] // 2, max(1, case["free"] // 10)

        def flanked(buf, off, ln, a):
            n2 = (ln + 2 * a).astype(np.int32)
            o2 = np.concatenate([[0], np.cumsum(n2[:-1], dtype=np.int64)]).astype(np.int64)
            out = np.frombuffer(b"ACGT", np.uint8)[r.integers(0, 4, int(n2.sum()) + 16)]
            src = np.repeat(off - np.concatenate([[0], np.cumsum(ln[:-1], dtype=np.int64)]), ln) + np.arange(int(ln.sum()))
            dst = np.repeat(o2 + a - np.concatenate([[0], np.cumsum(ln[:-1], dtype=np.int64)]), ln) + np.arange(int(ln.sum()))
            out[dst] = buf[src]
            return out, o2, n2

        pbuf, poff, plen = flanked(pbuf, poff, plen, g)
        tbuf, toff, tlen = flanked(tbuf, toff, tlen, f)
    return pbuf, poff, plen, tbuf, toff, tlen


def _run_room(case):
    """CIGAR runs a caller makes room for: two per edit, a half more, and some
    for the ends; the bases by the mean of the lengths and six standard
    deviations."""
    lo, hi, n = case["length"], case["max_length"], case["pairs"]
    mean = (hi - lo) / math.log(hi / lo) if hi > lo else hi
    bases = min(n * hi, n * mean + 6 * math.sqrt(n) * (hi - lo))
    return int(min(3 * case["max_rate"], 2) * bases + n * (4 * case["free"] + 40))


def _pinned(a):
    t = torch.empty(a.shape, dtype={"uint8": torch.uint8, "int32": torch.int32, "int64": torch.int64}[a.dtype.name],
                    pin_memory=True)
    t.numpy()[...] = a
    return t


def prepare(case, seed):
    b = _batch(case, seed)
    n, room = case["pairs"], _run_room(case)
    # a program that shares the GPU gives the engine a part of its memory
    al = T.Aligner(**MODELS[case["model"]][0], mem_budget=44 * GB)
    if case["free"]:
        al.set_ends_free(*([case["free"]] * 4))
    if case["option"] == "low_memory":
        al.set_low_memory(-1)
    st = {"al": al, "cigar": case["cigar"], "bidir": case["option"] == "bidirectional", "via": case["via"]}
    if case["via"] == "host":
        st["keep"] = [_pinned(x) for x in b]
        st["in"] = [t.numpy() for t in st["keep"]]
        outs = [_pinned(np.zeros(n, np.int32)), _pinned(np.zeros(n + 1, np.int64)), _pinned(np.zeros(room, np.int32))]
        st["keep"] += outs
        st["out"] = (outs[0].numpy(), outs[1].numpy(), outs[2].numpy().view(np.uint32))
        return st
    st["in"] = [torch.from_numpy(x).cuda() for x in b]
    st["scores"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    st["off"] = torch.zeros(n + 1, dtype=torch.int64, device="cuda") if case["cigar"] else None
    st["runs"] = torch.zeros(room, dtype=torch.int32, device="cuda") if case["cigar"] else None
    return st


def run(state):
    al, cigar, bidir = state["al"], state["cigar"], state["bidir"]
    if state["via"] == "host":
        scores, off, _ = al.align_arrays(*state["in"], cigar=cigar, out=state["out"], bidirectional=bidir)
        return [scores, off, state["out"][2].view(np.int32)] if cigar else [scores]
    p, po, pl, t, to, tl = state["in"]
    al.align_device(p, po, pl, t, to, tl, state["scores"], state["runs"], state["off"], bidirectional=bidir)
    return [state["scores"], state["off"], state["runs"]] if cigar else [state["scores"]]


def work(case):
    """Bytes: sequences, offsets and lengths read, scores (and offsets and
    runs: about two per edit) written.  Operations: the 9 additions, maxima
    and comparisons of a wavefront cell's recurrence (16 with two gap pieces,
    5 without an opening cost) and one extension test, for every cell of the
    narrowest exact search known (half of the full wavefronts)."""
    lengths, rates = _lengths(case, 1)
    edits = float(np.sum(lengths * rates))
    read = 2.0 * float(np.sum(lengths, dtype=np.float64)) + 2.4 * case["free"] * case["pairs"] / 2 + 24.0 * case["pairs"]
    wrote = 4.0 * case["pairs"] + (8.0 * case["pairs"] + 8.0 * edits if case["cigar"] else 0.0)
    per_cell = {"affine": 9, "dual": 16}.get(case["model"], 5) + 1
    return {"bytes": read + wrote, "flops": per_cell * 0.5 * _cells(case)}


def _affine_scores(b, x, o, e):
    """Gap-affine scores by dynamic programming over anti-diagonals in 64-bit
    integers, all pairs of a batch at once (lengths equal within a side)."""
    pbuf, poff, plen, tbuf, toff, tlen = b
    m, n, N = int(plen[0]), int(tlen[0]), len(plen)
    p = pbuf[poff[:, None] + np.arange(m)]
    t = tbuf[toff[:, None] + np.arange(n)]
    inf = np.int64(1) << 40

    def none():
        return np.full((N, m + 1), inf, np.int64)

    h2, h1, d1, i1 = none(), none(), none(), none()  # by row: H two and one anti-diagonals back, D and I one back
    h1[:, 0] = 0  # anti-diagonal 0
    for a in range(1, m + n + 1):
        lo, hi = max(0, a - n), min(m, a)
        h, d, i = none(), none(), none()
        r0, r1 = max(1, lo), hi  # rows with a cell above
        if r0 <= r1:
            d[:, r0:r1 + 1] = np.minimum(h1[:, r0 - 1:r1] + o + e, d1[:, r0 - 1:r1] + e)
        c1 = min(hi, a - 1)  # rows with a cell to the left
        if lo <= c1:
            i[:, lo:c1 + 1] = np.minimum(h1[:, lo:c1 + 1] + o + e, i1[:, lo:c1 + 1] + e)
        h[:, lo:hi + 1] = np.minimum(d[:, lo:hi + 1], i[:, lo:hi + 1])
        if r0 <= c1:
            rows = np.arange(r0, c1 + 1)
            sub = np.where(p[:, rows - 1] == t[:, a - rows - 1], 0, x)
            h[:, r0:c1 + 1] = np.minimum(h[:, r0:c1 + 1], h2[:, r0 - 1:c1] + sub)
        h2, h1, d1, i1 = h1, h, d, i
    return h1[:, m]


def exact(case, seed):
    """Scores of the small gap-affine cases; nothing in place of the CIGARs
    (several are optimal) and for the cases that would take minutes."""
    plain = case["model"] == "affine" and not case["free"] and case["length"] == case["max_length"]
    if not plain or case["pairs"] * float(case["length"]) ** 2 > 3e8:
        return None
    kw = MODELS["affine"][0]
    pbuf, poff, plen, tbuf, toff, tlen = _batch(case, seed)
    part = [slice(i, i + 250) for i in range(0, case["pairs"], 250)]  # a part's rows stay in cache
    scores = np.concatenate([_affine_scores((pbuf, poff[s], plen[s], tbuf, toff[s], tlen[s]), kw["mismatch"],
                                            kw["gap_opening"], kw["gap_extension"]) for s in part])
    return [scores, None, None] if case["cigar"] else [scores]
