"""The work that users of this framework have it do, as cases with seeded inputs.

A case is a dict of plain values.  ``listed()`` holds one case per kind of use, ``draw(rng)``
more cases of the same ranges, ``prepare(case, seed)`` what a program has in hand before the
call (inputs, configured aligner, result buffer), ``run(state)`` one pass through the public
entry points, ``work(case)`` the bytes and operations of a pass, and ``exact(case, seed)`` the
results in 64-bit integers from plain torch.

Scores follow the framework's sign convention: a gap of length k scores open + k * extension.
Sequences are synthetic: random DNA or protein, mutated copies with substitutions and
insertion / deletion runs, as the package's own workloads draw them (made here on the GPU, so
that a batch takes milliseconds).
"""
import math
import os

import numpy as np
import torch

import pairwise_aligner_gb300 as pa
from pairwise_aligner_gb300 import seqio
from pairwise_aligner_gb300.aligner import Aligner, Context

AMINO = b"ARNDCQEGHILKMFPSTWYV"
# BLOSUM62 over AMINO, row by row.
BLOSUM62 = [
    [4, -1, -2, -2, 0, -1, -1, 0, -2, -1, -1, -1, -1, -2, -1, 1, 0, -3, -2, 0],
    [-1, 5, 0, -2, -3, 1, 0, -2, 0, -3, -2, 2, -1, -3, -2, -1, -1, -3, -2, -3],
    [-2, 0, 6, 1, -3, 0, 0, 0, 1, -3, -3, 0, -2, -3, -2, 1, 0, -4, -2, -3],
    [-2, -2, 1, 6, -3, 0, 2, -1, -1, -3, -4, -1, -3, -3, -1, 0, -1, -4, -3, -3],
    [0, -3, -3, -3, 9, -3, -4, -3, -3, -1, -1, -3, -1, -2, -3, -1, -1, -2, -2, -1],
    [-1, 1, 0, 0, -3, 5, 2, -2, 0, -3, -2, 1, 0, -3, -1, 0, -1, -2, -1, -2],
    [-1, 0, 0, 2, -4, 2, 5, -2, 0, -3, -3, 1, -2, -3, -1, 0, -1, -3, -2, -2],
    [0, -2, 0, -1, -3, -2, -2, 6, -2, -4, -4, -2, -3, -3, -2, 0, -2, -2, -3, -3],
    [-2, 0, 1, -1, -3, 0, 0, -2, 8, -3, -3, -1, -2, -1, -2, -1, -2, -2, 2, -3],
    [-1, -3, -3, -3, -1, -3, -3, -4, -3, 4, 2, -3, 1, 0, -3, -2, -1, -3, -1, 3],
    [-1, -2, -3, -4, -1, -2, -3, -4, -3, 2, 4, -2, 2, 0, -3, -2, -1, -2, -1, 1],
    [-1, 2, 0, -1, -3, 1, 1, -2, -1, -3, -2, 5, -1, -3, -1, 0, -1, -3, -2, -2],
    [-1, -1, -2, -3, -1, 0, -2, -3, -2, 1, 2, -1, 5, 0, -2, -1, -1, -1, -1, 1],
    [-2, -3, -3, -3, -2, -3, -3, -3, -1, 0, 0, -3, 0, 6, -4, -2, -2, 1, 3, -1],
    [-1, -2, -2, -1, -3, -1, -1, -2, -2, -3, -3, -1, -2, -4, 7, -1, -1, -4, -3, -2],
    [1, -1, 1, 0, -1, 0, 0, 0, -1, -2, -2, 0, -1, -2, -1, 4, 1, -3, -2, -2],
    [0, -1, 0, -1, -1, -1, -1, -2, -2, -1, -1, -1, -1, -2, -1, 1, 5, -2, -2, 0],
    [-3, -3, -4, -4, -2, -2, -3, -2, -2, -3, -2, -3, -1, 1, -4, -3, -2, 11, 2, -3],
    [-2, -2, -2, -3, -2, -1, -2, -3, 2, -1, -1, -2, -1, 3, -3, -2, -2, 2, 7, -1],
    [0, -3, -3, -3, -1, -2, -2, -3, -3, 3, 1, -2, 1, -1, -2, -2, 0, -3, -1, 4],
]

# Per kind of use: scoring, end gaps and how the lengths are drawn.
KINDS = {
    # global alignment of short reads, small batches on the device: launches and latency count
    "reads": dict(match=2, mismatch=-3, open=-5, ext=-1),
    # a handful of pairs from host arrays: the smallest call a program makes
    "host_pairs": dict(match=4, mismatch=-5, open=-10, ext=-1),
    # local alignment of 64-512 bp fragments, half of them unrelated: the headline batch
    "local": dict(local=True, match=1, mismatch=-4, open=-6, ext=-1),
    # global alignment of fragments with structural indels
    "global_sv": dict(match=1, mismatch=-4, open=-6, ext=-1),
    # global alignment of long reads with log-normal lengths
    "long_reads": dict(match=2, mismatch=-4, open=-4, ext=-2),
    # a mixed stream: many short, some 1-10 kb and a few 20-50 kb global pairs
    "mixed": dict(match=1, mismatch=-4, open=-6, ext=-1),
    # the same stream with the learned band and its certificate
    "mixed_band": dict(match=1, mismatch=-4, open=-6, ext=-1, band_mode=1),
    # reads placed in longer reference windows: the window's ends are free; some reads hold an N
    "map_reads": dict(match=2, mismatch=-4, open=-4, ext=-2, first_column_free=True, last_column_free=True),
    # protein search: local alignment under BLOSUM62
    "protein": dict(local=True, open=-11, ext=-1, matrix=True),
    # alignment paths (begin, end, ops) of ~1 kb fragments, from and to host arrays
    "traceback": dict(match=2, mismatch=-4, open=-4, ext=-2),
    # local alignment of contigs of several kb; the scores of the longest pass 16 bits
    "contigs": dict(local=True, match=5, mismatch=-4, open=-10, ext=-1),
    # reads on the device into 2-bit words and into alphabet ranks
    "encode": dict(),
}


def listed():
    return [
        {"name": "reads_1k", "kind": "reads", "pairs": 1024, "lo": 150, "hi": 150},
        {"name": "host_16_pairs", "kind": "host_pairs", "pairs": 16, "lo": 80, "hi": 400},
        {"name": "local_262k", "kind": "local", "pairs": 262144, "lo": 64, "hi": 512},
        {"name": "global_sv_16k", "kind": "global_sv", "pairs": 16384, "lo": 64, "hi": 512},
        {"name": "long_reads_4k", "kind": "long_reads", "pairs": 4001, "lo": 500, "hi": 20000},
        {"name": "mixed_33k", "kind": "mixed", "pairs": 32768, "lo": 100, "hi": 50000},
        {"name": "mixed_band_33k", "kind": "mixed_band", "pairs": 32768, "lo": 100, "hi": 50000},
        {"name": "map_reads_65k", "kind": "map_reads", "pairs": 65537, "lo": 100, "hi": 250},
        {"name": "protein_33k", "kind": "protein", "pairs": 32768, "lo": 50, "hi": 1000},
        {"name": "traceback_4k", "kind": "traceback", "pairs": 4096, "lo": 500, "hi": 2000},
        {"name": "contigs_500", "kind": "contigs", "pairs": 500, "lo": 2000, "hi": 20000},
        {"name": "encode_256M", "kind": "encode", "pairs": 1789570, "lo": 100, "hi": 200},
    ]


# How far drawn cases of a kind spread: pairs, shortest and longest length.
RANGES = {
    "reads": ((200, 5000), (90, 150), (150, 260)),
    "host_pairs": ((1, 64), (40, 200), (200, 500)),
    "local": ((6000, 262144), (48, 96), (300, 512)),
    "global_sv": ((3000, 33000), (64, 128), (300, 512)),
    "long_reads": ((600, 4100), (500, 800), (12000, 20000)),
    "mixed": ((5000, 33000), (100, 100), (50000, 50000)),
    "mixed_band": ((5000, 33000), (100, 100), (50000, 50000)),
    "map_reads": ((8000, 100000), (75, 120), (151, 250)),
    "protein": ((4000, 33000), (40, 80), (600, 1000)),
    "traceback": ((700, 4100), (300, 600), (1200, 2000)),
    "contigs": ((90, 510), (1500, 2500), (8000, 20000)),
    "encode": ((60000, 1789570), (90, 110), (150, 250)),
}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(sorted(KINDS))
    pairs, lo, hi = RANGES[kind]
    return {"kind": kind, "pairs": _log_uniform(rng, *pairs), "lo": _log_uniform(rng, *lo),
            "hi": _log_uniform(rng, *hi)}


# ---- seeded sequences, on the GPU -------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _offsets(lens):
    off = torch.zeros(lens.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=off[1:])
    return off


def _uniform_lengths(g, n, lo, hi):
    return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda")


def _log_normal_lengths(g, n, median, sigma, lo, hi):
    x = torch.exp(math.log(median) + sigma * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    return x.round().long().clamp(lo, hi)


def _random(g, total, symbols):
    return torch.randint(0, symbols, (total,), generator=g, device="cuda", dtype=torch.uint8)


def _mutate(g, codes, off, p_sub, p_ins, p_del, mean, symbols):
    """Per base: a deletion run starts, an insertion run is placed before it, or it is replaced
    by another symbol; runs have geometric lengths of the given mean.  -> (codes, offsets)."""
    n = codes.numel()

    def run_lengths():
        if mean <= 1.0:
            return torch.ones(n, dtype=torch.int64, device="cuda")
        u = torch.rand(n, generator=g, device="cuda").clamp_min(1e-9)
        return 1 + torch.floor(torch.log(u) / math.log(1.0 - 1.0 / mean)).long()

    u = torch.rand(n, generator=g, device="cuda")
    pair = torch.repeat_interleave(torch.arange(off.numel() - 1, device="cuda"), off[1:] - off[:-1])
    pos = torch.arange(n, device="cuda")
    start = u < p_del
    # the furthest end of a deletion run that started at or before a base, within its pair
    end = torch.where(start, torch.minimum(pos + run_lengths(), off[1:][pair]), torch.zeros_like(pos))
    deleted = torch.cummax(end, 0).values > pos
    sub = (u >= p_del) & (u < p_del + p_sub)
    shift = torch.randint(1, symbols, (n,), generator=g, device="cuda", dtype=torch.uint8)
    base = torch.where(sub, (codes + shift) % symbols, codes)
    ins = torch.where(torch.rand(n, generator=g, device="cuda") < p_ins, run_lengths(), torch.zeros_like(pos))
    counts = ins + (~deleted).long()
    src = torch.repeat_interleave(pos, counts)
    first = torch.cumsum(counts, 0) - counts
    rank = torch.arange(src.numel(), device="cuda") - first[src]
    fresh = torch.randint(0, symbols, (src.numel(),), generator=g, device="cuda", dtype=torch.uint8)
    out = torch.where(rank < ins[src], fresh, base[src])
    total = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(counts, 0)])
    return out, total[off]


def _window(g, codes, off, target, symbols):
    """Crop every sequence to a random window of target bases, or pad it with random flanks."""
    lens = off[1:] - off[:-1]
    shift = (torch.rand(lens.numel(), generator=g, device="cuda") * ((lens - target).abs() + 1)).long()
    shift = torch.where(lens >= target, shift, -shift)
    new = _offsets(target)
    pair = torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), target)
    pos = torch.arange(int(new[-1]), device="cuda") - new[pair] + shift[pair]
    inside = (pos >= 0) & (pos < lens[pair])
    src = (off[pair] + pos.clamp_min(0)).clamp_max(max(codes.numel() - 1, 0))
    fresh = _random(g, pos.numel(), symbols)
    return torch.where(inside, codes[src], fresh), new


def _structural(g, codes, off, symbols, lo=50, hi=500):
    """One deletion or insertion run of lo..hi bases per sequence, at a random place."""
    n_pairs = off.numel() - 1
    lens = off[1:] - off[:-1]
    run = torch.randint(lo, hi + 1, (n_pairs,), generator=g, device="cuda")
    at = (torch.rand(n_pairs, generator=g, device="cuda") * (lens + 1)).long()
    grow = torch.rand(n_pairs, generator=g, device="cuda") < 0.5
    cut = torch.where(grow, -run, torch.minimum(run, (lens - at).clamp_min(0)))
    new = _offsets(lens - cut)
    pair = torch.repeat_interleave(torch.arange(n_pairs, device="cuda"), lens - cut)
    pos = torch.arange(int(new[-1]), device="cuda") - new[pair]
    a, c = at[pair], cut[pair]
    fresh_at = (c < 0) & (pos >= a) & (pos < a - c)
    src = torch.where(pos < a, pos, pos + c)
    src = torch.where(fresh_at, torch.zeros_like(src), src)
    fresh = _random(g, pos.numel(), symbols)
    return torch.where(fresh_at, fresh, codes[(off[pair] + src).clamp_max(max(codes.numel() - 1, 0))]), new


def _interleave(parts, n):
    """Pairs of several groups (codes, offsets, pair ids) merged into pair order."""
    lens = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _, off, idx in parts:
        lens[idx] = off[1:] - off[:-1]
    new = _offsets(lens)
    out = torch.empty(int(new[-1]), dtype=torch.uint8, device="cuda")
    for codes, off, idx in parts:
        shift = torch.repeat_interleave(new[idx] - off[:-1], off[1:] - off[:-1])
        out[shift + torch.arange(codes.numel(), device="cuda")] = codes
    return out, new


def _sequences(case, seed):
    """The batch of a case: (codes1, off1, codes2, off2, symbols); codes index the alphabet, and
    a code equal to `symbols` is an N."""
    g, kind, n, lo, hi = _gen(seed), case["kind"], case["pairs"], case["lo"], case["hi"]
    if kind == "encode":
        codes = _random(g, n * (lo + hi) // 2, 4)
        codes[torch.rand(codes.numel(), generator=g, device="cuda") < 1e-3] = 4
        return codes, None, None, None, 4
    if kind in ("mixed", "mixed_band"):
        # 90 % of lo..300 bp at 10 %, 9 % of 1-10 kb at 8 %, 1 % of 20-50 kb at 6 % divergence
        u = torch.rand(n, generator=g, device="cuda")
        p1, p2 = [], []
        for sel, a, b, div, sv in ((u < 0.90, lo, 300, 0.10, False), ((u >= 0.90) & (u < 0.99), 1000, 10000, 0.08, False),
                                   (u >= 0.99, 20000, hi, 0.06, True)):
            idx = torch.nonzero(sel).flatten()
            if idx.numel() == 0:
                continue
            off = _offsets(_uniform_lengths(g, idx.numel(), a, b))
            q = _random(g, int(off[-1]), 4)
            t, toff = _mutate(g, q, off, 0.8 * div, 0.1 * div, 0.1 * div, 2.0, 4)
            if sv:
                t, toff = _structural(g, t, toff, 4)
            p1.append((q, off, idx))
            p2.append((t, toff, idx))
        return _interleave(p1, n) + _interleave(p2, n) + (4,)
    if kind == "map_reads":
        # the window (sequence1) holds the read's template plus flanks of up to one read length
        lens = _uniform_lengths(g, n, lo, hi)
        off = _offsets(lens)
        q = _random(g, int(off[-1]), 4)
        t, toff = _mutate(g, q, off, 0.02, 0.005, 0.005, 1.5, 4)
        w, woff = _window(g, q, off, lens + (torch.rand(n, generator=g, device="cuda") * lens).long() + 20, 4)
        with_n = torch.nonzero(torch.rand(n, generator=g, device="cuda") < 0.01).flatten()
        t[(toff[with_n] + (toff[with_n + 1] - toff[with_n]) // 2).clamp_max(t.numel() - 1)] = 4
        return w, woff, t, toff, 4
    if kind == "protein":
        lens = _log_normal_lengths(g, n, 280.0, 0.6, lo, hi)
        off = _offsets(lens)
        q = _random(g, int(off[-1]), 20)
        t, toff = _mutate(g, q, off, 0.5, 0.02, 0.02, 2.0, 20)
        t, toff = _window(g, t, toff, _log_normal_lengths(g, n, 280.0, 0.6, lo, hi), 20)
        u, uoff = _random(g, t.numel(), 20), toff
        related = torch.rand(n, generator=g, device="cuda") < 0.2
        pair = torch.repeat_interleave(torch.arange(n, device="cuda"), uoff[1:] - uoff[:-1])
        return q, off, torch.where(related[pair], t, u), toff, 20
    if kind == "long_reads":
        off = _offsets(_log_normal_lengths(g, n, 3000.0, 0.6, lo, hi))
    elif kind == "contigs":
        off = _offsets(_log_normal_lengths(g, n, 6000.0, 0.5, lo, hi))
    else:
        # the op buffer is as long as the sequences: its size is the case's, not the seed's
        off = _offsets(_uniform_lengths(_gen(n) if kind == "traceback" else g, n, lo, hi))
    q = _random(g, int(off[-1]), 4)
    rates = {"reads": (0.08, 0.01, 0.01, 2.0), "host_pairs": (0.08, 0.01, 0.01, 2.0), "local": (0.15, 0.02, 0.02, 2.0),
             "global_sv": (0.15, 0.02, 0.02, 2.0), "long_reads": (0.05, 0.03, 0.03, 1.5),
             "traceback": (0.06, 0.02, 0.02, 1.5), "contigs": (0.05, 0.01, 0.01, 2.0)}[kind]
    t, toff = _mutate(g, q, off, *rates, 4)
    if kind == "global_sv":
        t, toff = _structural(g, t, toff, 4)
    if kind == "traceback":
        t, toff = _window(g, t, toff, off[1:] - off[:-1], 4)
    if kind in ("local", "contigs"):
        # sequence2 is a window of its own length; half of the local fragments are unrelated
        target = (_uniform_lengths(g, n, lo, hi) if kind == "local"
                  else _log_normal_lengths(g, n, 6000.0, 0.5, lo, hi))
        t, toff = _window(g, t, toff, target, 4)
        if kind == "local":
            pair = torch.repeat_interleave(torch.arange(n, device="cuda"), target)
            related = torch.rand(n, generator=g, device="cuda") < 0.5
            t = torch.where(related[pair], t, _random(g, t.numel(), 4))
    return q, off, t, toff, 4


def _letters(codes, symbols):
    table = torch.tensor(list(b"ACGTN" if symbols == 4 else AMINO), dtype=torch.uint8, device="cuda")
    return table[codes.long()]


def _config(kind):
    k = KINDS[kind]
    local = bool(k.get("local"))
    conf = dict(local=local, match=k.get("match", 0), mismatch=k.get("mismatch", 0), gap_open=k["open"],
                gap_extension=k["ext"], first_column_free=local or bool(k.get("first_column_free")),
                first_row_free=local, last_column_free=local or bool(k.get("last_column_free")), last_row_free=local,
                width_hint=0, band_mode=k.get("band_mode", 0))
    if k.get("matrix"):
        conf["matrix"] = (AMINO, tuple(x for row in BLOSUM62 for x in row))
    return conf


# ---- one pass --------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    q, off1, t, off2, symbols = _sequences(case, seed)
    s1 = _letters(q, symbols)
    if kind == "encode":
        n = s1.numel()
        state = dict(kind=kind, ctx=Context(0), s1=s1, words=torch.empty((n + 15) // 16, dtype=torch.int32, device="cuda"),
                     ranks=torch.empty(n, dtype=torch.int8, device="cuda"))
    else:
        s2 = _letters(t, symbols)
        aligner = Aligner(_config(kind), context=Context(0))
        if kind == "mixed_band":
            path = os.path.join(os.path.dirname(pa.__file__), "data", "band_model.npz")
            with np.load(path) as z:
                aligner.context.set_band_model({k: z[k] for k in z.files})
        state = dict(kind=kind, aligner=aligner)
        if kind in ("host_pairs", "traceback"):
            state.update(s1=s1.cpu().numpy(), o1=off1.cpu().numpy().astype(np.uint64), s2=s2.cpu().numpy(),
                         o2=off2.cpu().numpy().astype(np.uint64))
        else:
            state.update(s1=s1, o1=off1, s2=s2, o2=off2,
                         out=torch.zeros((case["pairs"], 4), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "encode":
        seqio.pack_2bit_device(state["ctx"], state["s1"], state["words"])
        seqio.rank_map_device(state["ctx"], b"ACGTN", state["s1"], state["ranks"])
        return state["words"], state["ranks"]
    args = state["s1"], state["o1"], state["s2"], state["o2"]
    if kind == "host_pairs":
        res = state["aligner"].compute_arrays(*args)
        return res["score"], res["end1"], res["end2"], res["width"], res["flags"]
    if kind == "traceback":
        res, aln, ops, ops_off = state["aligner"].compute_traceback_arrays(*args)
        # a pair's region holds n_ops ops; what follows them in it means nothing
        used = aln["n_ops"].astype(np.int64)
        room = np.diff(np.append(ops_off, np.uint64(len(ops))).astype(np.int64))
        keep = np.repeat(np.tile(np.array([255, 0], np.uint8), len(used)), np.stack([used, room - used], 1).ravel())
        np.bitwise_and(ops, keep, out=ops)
        return res["score"], res["end1"], res["end2"], aln["begin1"], aln["begin2"], aln["n_ops"], ops
    out = state["out"]
    state["aligner"].compute_device(*args, out, stream=torch.cuda.current_stream())
    # score, end in sequence1, end in sequence2, and width | flags | band rounds in one word
    return out[:, 0], out[:, 1], out[:, 2], out[:, 3]


def _mean_lengths(case):
    """Expected m + n and m * n of a pair."""
    lo, hi, kind = case["lo"], case["hi"], case["kind"]
    mid, var = (lo + hi) / 2.0, (hi - lo) ** 2 / 12.0
    if kind in ("mixed", "mixed_band"):
        parts = ((0.90, lo, 300), (0.09, 1000, 10000), (0.01, 20000, hi))
        return (sum(2 * p * (a + b) / 2.0 for p, a, b in parts),
                sum(p * (((a + b) / 2.0) ** 2 + (b - a) ** 2 / 12.0) for p, a, b in parts))
    if kind in ("long_reads", "contigs", "protein"):
        median, sigma = {"long_reads": (3000.0, 0.6), "contigs": (6000.0, 0.5), "protein": (280.0, 0.6)}[kind]
        mean = median * math.exp(sigma * sigma / 2)
        return 2 * mean, mean * mean * (math.exp(sigma * sigma) if kind == "long_reads" else 1.0)
    if kind == "map_reads":
        return 2.5 * mid + 20, 1.5 * (mid * mid + var) + 20 * mid
    if kind == "local":
        return 2 * mid, mid * mid
    return 2 * mid, mid * mid + var


def work(case):
    """Sequences and offsets read once, results written once; per DP cell the five maxima and
    adds of the affine recurrence count as 5 operations."""
    n, kind = case["pairs"], case["kind"]
    if kind == "encode":
        bases = n * (case["lo"] + case["hi"]) // 2
        return {"bytes": int(bases * 2.25), "flops": 0}     # read once; a quarter byte and a rank each
    sum_len, cells = _mean_lengths(case)
    total = n * (sum_len + 16 + 16)
    if kind == "traceback":
        total += n * (16 + sum_len / 2)
    return {"bytes": int(total), "flops": int(5 * n * cells)}


# ---- the results in 64-bit integers -------------------------------------------------------------
def _padded(codes, off, fill):
    lens = off[1:] - off[:-1]
    pos = torch.arange(int(lens.max()), device="cuda")[None, :]
    idx = (off[:-1, None] + pos).clamp_max(codes.numel() - 1)
    return torch.where(pos < lens[:, None], codes[idx].long(), torch.full_like(idx, fill)), lens


def _dp(a, m, b, n, score_of, conf):
    """Affine-gap scores and end cells of padded batches, column by column in int64: among equal
    scores the smallest end in sequence1, then in sequence2, wins."""
    lowest = -(1 << 40)
    go, ge, local = conf["gap_open"], conf["gap_extension"], conf["local"]
    rows = b.shape[1]
    j = torch.arange(rows + 1, device="cuda")
    border = torch.where(j > 0, go + ge * j, torch.zeros_like(j))
    first = torch.zeros_like(border) if conf["first_row_free"] else border
    h = first[None, :].expand(a.shape[0], -1).contiguous()
    gap = h + go + ge
    valid = j[None, :] <= n[:, None]
    is_n = j[None, :] == n[:, None]
    best = torch.full_like(m, 0 if local else lowest)
    e1, e2 = torch.zeros_like(m), torch.zeros_like(m)

    def offer(x, i, take):
        nonlocal best, e1, e2
        v, jj = torch.where(take, x, torch.full_like(x, lowest)).max(1)
        jj = (torch.where(take, x, torch.full_like(x, lowest)) == v[:, None]).long().argmax(1)
        up = v > best
        best, e1, e2 = torch.where(up, v, best), torch.where(up, torch.full_like(e1, i), e1), torch.where(up, jj, e2)

    if not local and conf["last_column_free"]:
        offer(h, 0, is_n)
    for i in range(1, a.shape[1] + 1):
        x = h[:, :-1] + score_of(a[:, i - 1], b)
        if local:
            x = x.clamp_min_(0)
        x = torch.maximum(x, gap[:, 1:])
        top = 0 if conf["first_column_free"] else go + ge * i
        x = torch.cat([torch.full_like(x[:, :1], top), x], 1)
        run = torch.cummax(x - ge * j, 1).values
        h = x
        h[:, 1:] = torch.maximum(x[:, 1:], run[:, :-1] + go + ge * j[1:])
        gap = torch.maximum(gap + ge, h + go + ge)
        inside = (i <= m)[:, None]
        if local:
            offer(h, i, valid & inside & (j > 0))
        else:
            take = is_n & (i == m)[:, None]
            if conf["last_column_free"]:
                take = take | (is_n & inside)
            if conf["last_row_free"]:
                take = take | (valid & (i == m)[:, None])
            offer(h, i, take)
    if local:
        e1, e2 = torch.where(best > 0, e1, 0), torch.where(best > 0, e2, 0)
    return best, e1, e2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixed", "mixed_band", "long_reads", "contigs"):
        return None                       # minutes in 64 bits
    q, off1, t, off2, symbols = _sequences(case, seed)
    if kind == "encode":
        code = torch.where(q == 4, torch.tensor((ord("N") >> 1 ^ ord("N") >> 2) & 3, device="cuda"), q.long())
        code = torch.nn.functional.pad(code, (0, -code.numel() % 16)).view(-1, 16)
        words = (code << (2 * torch.arange(16, device="cuda"))).sum(1)
        return torch.where(words >= 1 << 31, words - (1 << 32), words), q.long()
    conf = _config(kind)
    if symbols == 4:
        def score_of(x, y):
            return torch.where(x[:, None] == y, conf["match"], conf["mismatch"])
    else:
        table = torch.nn.functional.pad(torch.tensor(BLOSUM62, device="cuda"), (0, 2, 0, 2), value=-9).contiguous()

        def score_of(x, y):
            return table[x[:, None], y]
    step = max(1, int(2e8 // (case["hi"] * 3)))
    parts = []
    for k in range(0, case["pairs"], step):
        e = min(k + step, case["pairs"])
        a, m = _padded(q, off1[k:e + 1], 21 if symbols == 20 else 6)
        b, n = _padded(t, off2[k:e + 1], 20 if symbols == 20 else 7)
        parts.append(_dp(a, m, b, n, score_of, conf))
    score, e1, e2 = (torch.cat(p) for p in zip(*parts))
    if kind == "traceback":
        return score, e1, e2, None, None, None, None
    if kind == "host_pairs":
        return score, e1, e2, None, None
    return score, e1, e2, None
