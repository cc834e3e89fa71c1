"""The measured workloads of the seed-and-filter path.

Each case is one pass of what a program built on this package does with it:
one seed_and_filter call, a plain pass over a query, many query blocks in one
batched pass, a unit from ASCII bases to records, a burst of served requests,
or the dedup of HSPs that already sit in device memory.  Sizes follow the
package's own workloads (1 Mbp pairs, 10 Mbp target bins, 250 kbp calls, 10
kbp - 2 Mbp query chunks against a resident 200 Mbp target, repeat-dense pairs
with an occurrence cap, lognormal requests); sequences have their composition:
41 % GC, 10 % soft-masked runs, planted homology.
"""
from __future__ import annotations

import ctypes as C
import os
import tempfile

import numpy as np
import torch

from hspz_b200 import Engine, EngineConfig, build_sub_mat
from hspz_b200 import _native as N
from hspz_b200 import synth
from hspz_b200.hsp import SEGMENT_PAIR

# A LASTZ score set for close species.  Its mismatches do not fit a signed
# byte, unlike the default matrix's.
CLOSE_SPECIES = """# close species
bad_score = X:-1000
fill_score = -100
     A    C    G    T
A   90 -330 -236 -356
C -330  100 -318 -236
G -236 -318  100 -330
T -356 -236 -330   90
"""

# kind, target bases, total query bases, query blocks, seed, transitions,
# occurrence cap, matrix: "default" or "close", strand
_LISTED = [
    # The smallest call: the reference's engine works through a query in calls
    # of 250 kbp, here one call against one 10 Mbp target bin.
    dict(name="call_250k", kind="call", target=10_000_000, query=250_019, blocks=1),
    # A small pair of sequences (bacterial genomes, BACs): upload and one plain
    # pass, a few calls with little work each.
    dict(name="pass_1m", kind="swap_pass", target=1_000_000, query=1_000_000, blocks=1),
    # The unit of a whole-genome run: one 10 Mbp bin against 10 Mbp of query.
    dict(name="pass_bin_10m", kind="pass", target=10_000_000, query=10_000_000, blocks=1),
    # The longer seed, on one strand, without the entropy test.
    dict(name="pass_14of22", kind="pass", target=50_000_000, query=3_000_001, blocks=1, seed="14of22",
         strand="plus", noentropy=True),
    # A score set for close species: mismatches wider than a byte.
    dict(name="pass_close_species", kind="pass", target=10_000_000, query=4_000_000, blocks=1, matrix="close"),
    # Many small contigs against a mid-sized target, exact seeds only.
    dict(name="batch_contigs", kind="batched", target=40_000_003, query=6_000_000, blocks=96, transitions=False),
    # The throughput workload: chunks of uneven length against a resident 200
    # Mbp target.
    dict(name="batch_chunks", kind="batched", target=200_000_000, query=16_000_000, blocks=48),
    # Repeat-dense sequences with an occurrence cap: long extensions, and many
    # more HSPs per base.
    dict(name="batch_repeats", kind="repeats", target=16_000_000, query=4_000_000, blocks=4, occ_cap=1000),
    # From ASCII to records: the seed table is built, the query staged, the
    # pass run (a program does this once per target bin).
    dict(name="unit_ascii", kind="unit", target=20_000_000, query=1_500_000, blocks=3),
    # A burst of requests to the serving loop over a resident target.
    dict(name="serve_burst", kind="serve", target=100_000_000, query=3_000_000, blocks=12),
    # Dedup of HSPs in the caller's device memory.
    dict(name="dedup_device", kind="dedup", records=200_003),
]

_DEFAULTS = dict(target=0, query=0, blocks=1, seed="12of19", transitions=True, occ_cap=0, matrix="default",
                 strand="both", noentropy=False, records=0)


def _full(case):
    return {**_DEFAULTS, **case}


def listed():
    return [_full(c) for c in _LISTED]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["call", "swap_pass", "pass", "pass_long_seed", "pass_close", "batched", "batched_exact",
                       "repeats", "unit", "serve", "dedup"])
    if kind == "call":
        return _full(dict(kind="call", target=_log(rng, 1_000_000, 100_000_000), query=_log(rng, 20_000, 250_019)))
    if kind == "swap_pass":
        return _full(dict(kind="swap_pass", target=_log(rng, 300_000, 5_000_000),
                          query=_log(rng, 300_000, 5_000_000), strand=rng.choice(["both", "plus", "minus"])))
    if kind == "pass":
        return _full(dict(kind="pass", target=_log(rng, 5_000_000, 40_000_000),
                          query=_log(rng, 1_000_000, 10_000_000), noentropy=rng.random() < 0.25))
    if kind == "pass_long_seed":
        return _full(dict(kind="pass", target=_log(rng, 10_000_000, 80_000_000),
                          query=_log(rng, 500_000, 5_000_000), seed="14of22",
                          strand=rng.choice(["both", "plus", "minus"]), transitions=rng.random() < 0.75))
    if kind == "pass_close":
        return _full(dict(kind="pass", target=_log(rng, 2_000_000, 20_000_000),
                          query=_log(rng, 500_000, 5_000_000), matrix="close"))
    if kind == "batched":
        return _full(dict(kind="batched", target=_log(rng, 20_000_000, 200_000_000),
                          query=_log(rng, 2_000_000, 16_000_000), blocks=_log(rng, 8, 100)))
    if kind == "batched_exact":
        return _full(dict(kind="batched", target=_log(rng, 20_000_000, 200_000_000),
                          query=_log(rng, 2_000_000, 16_000_000), blocks=_log(rng, 8, 100), transitions=False))
    if kind == "repeats":
        return _full(dict(kind="repeats", target=_log(rng, 4_000_000, 16_000_000),
                          query=_log(rng, 500_000, 4_000_000), blocks=rng.randrange(1, 7),
                          occ_cap=rng.choice([50, 200, 1000])))
    if kind == "unit":
        return _full(dict(kind="unit", target=_log(rng, 2_000_000, 40_000_000),
                          query=_log(rng, 200_000, 3_000_000), blocks=rng.randrange(1, 6)))
    if kind == "serve":
        return _full(dict(kind="serve", target=_log(rng, 30_000_000, 200_000_000),
                          query=_log(rng, 500_000, 4_000_000), blocks=rng.randrange(2, 17)))
    return _full(dict(kind="dedup", records=_log(rng, 1_000, 262_144)))


# --- inputs -------------------------------------------------------------------

def _bases(gen, n):
    """n random bases at 41 % GC."""
    lut = torch.from_numpy(np.repeat(synth.BASES, [59, 41, 41, 59]).copy()).cuda()
    return lut[torch.randint(0, 200, (n,), generator=gen, device="cuda", dtype=torch.uint8).int()].cpu().numpy()


def _soft_mask(rng, s):
    """Lowercase runs of 50-500 bp over ~10 % of s, in place."""
    k = int(s.size * 0.10 / 275) + 1
    starts = rng.integers(0, s.size, k)
    lens = rng.integers(50, 501, k)
    for a, n in zip(starts.tolist(), lens.tolist()):
        s[a:a + n] |= 0x20
    return s


def _block_lengths(rng, total, blocks):
    """Uneven block lengths (log-uniform over a factor of 200) of `total` bases in all."""
    w = np.exp(rng.uniform(0.0, np.log(200.0), blocks))
    return np.maximum((w / w.sum() * total).astype(np.int64), 1000 if total >= 1000 * blocks else 1)


def _sequences(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "repeats":
        fam = synth.repeat_families(rng)
        t = synth.repeat_genome(rng, case["target"], fam)
        q = synth.repeat_genome(rng, case["query"], fam)
        cuts = np.linspace(0, q.size, case["blocks"] + 1).astype(np.int64)
        queries = [q[a:b].copy() for a, b in zip(cuts[:-1], cuts[1:])]
        share = 0.05
    else:
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        t = _bases(gen, case["target"])
        lens = ([case["query"]] if case["blocks"] == 1
                else _block_lengths(rng, case["query"], case["blocks"]).tolist())
        queries = [_bases(gen, int(n)) for n in lens]
        share = 0.2
    for q in queries:
        synth.plant(rng, t, q, int(q.size * share / 2600), 200, 5000, 0.05, 0.35)
        _soft_mask(rng, q)
    return _soft_mask(rng, t), queries


def _config(case):
    if case["matrix"] == "close":
        fd, path = tempfile.mkstemp(suffix=".q")
        try:
            with os.fdopen(fd, "w") as f:
                f.write(CLOSE_SPECIES)
            sub_mat = build_sub_mat("", 910, path)
        finally:
            os.unlink(path)
    else:
        sub_mat = build_sub_mat("", 910)
    return EngineConfig(sub_mat=sub_mat, seed=case["seed"], transitions=case["transitions"],
                        occ_cap=case["occ_cap"], strand=case["strand"], noentropy=case["noentropy"])


def _hsp_records(case, seed):
    """HSPs as a pass leaves them: many overlap on shared diagonals."""
    rng = np.random.default_rng(seed)
    n = case["records"]
    a = np.zeros(n, dtype=SEGMENT_PAIR)
    a["query_start"] = rng.integers(0, 5_000_000, n)
    a["ref_start"] = a["query_start"] + rng.integers(0, 200_000_000, n).astype(np.uint32)
    a["len"] = rng.integers(40, 600, n)
    a["score"] = rng.integers(3000, 30000, n)
    src = rng.integers(0, n, n // 2)
    dst = rng.integers(0, n, n // 2)
    a[dst] = a[src]  # the same HSP found from another of its seeds, some of them cut short
    a["len"][dst[::3]] //= 2
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dedup":
        recs = _hsp_records(case, seed)
        d_in = torch.from_numpy(recs.view(np.uint8).copy()).cuda()
        return dict(case=case, d_in=d_in, n=case["records"], d_out=torch.zeros_like(d_in),
                    d_n=torch.zeros(1, dtype=torch.int32, device="cuda"))
    target, queries = _sequences(case, seed)
    e = Engine(_config(case))
    state = dict(case=case, engine=e, target=target, queries=queries)
    # the program's own array for a pass's records, with room to spare
    state["rows"] = np.zeros((case["query"] // (4 if kind == "repeats" else 64) + 256, 4 if kind == "call" else
                              6 if kind in ("swap_pass", "pass", "serve") else 7), dtype=np.int32)
    state["used"] = 0
    if kind != "unit":
        e.load_target(target)
    if kind in ("call", "pass"):
        e.swap_query_ascii(queries[0])
    elif kind in ("batched", "repeats"):
        e.stage_queries(queries)
    elif kind == "serve":
        e.serve_start(budget_bytes=16 << 30, workers=2)
    return state


# --- one pass -----------------------------------------------------------------

_COUNTS = ("seeds", "hits", "cells", "raw_hsps", "hsps", "calls")


def _keep(state, recs, at=0):
    """Puts records, as rows of 32-bit words, into the program's array at row `at`; returns the next row."""
    rows = state["rows"]
    if at + recs.size > len(rows):
        raise ValueError(f"{at + recs.size} records, room for {len(rows)}")
    rows[at:at + recs.size] = recs.view(np.int32).reshape(recs.size, rows.shape[1])
    return at + recs.size


def _done(state, end, counts):
    state["rows"][end:state["used"]] = 0  # rows of a longer pass before
    state["used"] = end
    return state["rows"], counts


def _out(state, result):
    recs, stats = result
    return _done(state, _keep(state, recs), [int(stats[k]) for k in _COUNTS])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dedup":
        N.check(N.lib().hz_dedup_and_order_device_noalloc(
            C.c_void_p(state["d_in"].data_ptr()), state["n"], C.c_void_p(state["d_out"].data_ptr()),
            C.c_void_p(state["d_n"].data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["d_out"], state["d_n"]
    e = state["engine"]
    if kind == "call":
        # the last base of the query ends the last seed window
        e.generate_seeds(0, False, (0, case["query"] - e.seed_size + 1))
        return _out(state, e.seed_and_filter(0, False))
    if kind == "pass":
        return _out(state, e.run_pass())
    if kind == "swap_pass":
        e.swap_query_ascii(state["queries"][0])
        return _out(state, e.run_pass())
    if kind in ("batched", "repeats"):
        return _out(state, e.run_batched())
    if kind == "unit":
        e.load_target(state["target"])
        e.stage_queries(state["queries"])
        return _out(state, e.run_batched())
    tickets = [e.serve_submit(q) for q in state["queries"]]
    end, ends = 0, []
    for t in tickets:
        end = _keep(state, e.serve_poll(t)[0], end)
        ends.append(end)
    return _done(state, end, ends)


# --- the least work -------------------------------------------------------------

_P = (0.295, 0.205, 0.205, 0.295)
_MATCH = sum(p * p for p in _P)           # two random bases are equal
_TRANSITION = 4 * _P[0] * _P[1]           # or differ by a transition
_UNMASKED = 0.9


def _expected_hits(case):
    """Seed hits of random sequences of this composition."""
    care, width = (14, 22) if case["seed"] == "14of22" else (12, 19)
    seeds = _MATCH ** care
    if case["transitions"]:
        seeds += care * _TRANSITION * _MATCH ** (care - 1)
    strands = 2 if case["strand"] == "both" and case["kind"] != "call" else 1
    return strands * case["query"] * case["target"] * _UNMASKED ** 2 * seeds


def work(case):
    if case["kind"] == "dedup":
        n = case["records"]
        # records in, kept records out; two sorts' comparisons
        return {"bytes": 16 * n + 12 * n, "flops": 2 * n * max(1, n.bit_length())}
    hits = _expected_hits(case)
    # Each base of both sequences once at 3 bits (2-bit code, mask bit), the
    # seed table's words that the pass looks at, each position word that hits
    # name; ~64 cells per hit with an add, a maximum and a drop test each.
    care = 14 if case["seed"] == "14of22" else 12
    strands = 2 if case["strand"] == "both" and case["kind"] != "call" else 1
    lookups = strands * case["query"] * (1 + care if case["transitions"] else 1)
    seq = 0.375 * (case["target"] + strands * case["query"])
    table = 4 * min(4 ** care, 2 * lookups) + 4 * min(case["target"], hits)
    ascii_in = case["target"] + case["query"] if case["kind"] == "unit" else (
        case["query"] if case["kind"] in ("swap_pass", "serve") else 0)
    return {"bytes": int(seq + table + ascii_in), "flops": int(3 * 64 * hits)}


# --- the exact answer -----------------------------------------------------------

def exact(case, seed):
    """Dedup restated in numpy: sort by (diagonal, start, length, score
    descending), drop a record contained in the one before it, sort by (query
    start, start, length, score descending).  The passes over sequences return
    whole numbers only, and are restated elsewhere as a program that takes
    minutes at these sizes."""
    if case["kind"] != "dedup":
        return None
    a = _hsp_records(case, seed)
    r, q, n, s = (a[f].astype(np.int64) for f in ("ref_start", "query_start", "len", "score"))
    diag = (r - q) & 0xFFFFFFFF
    o = np.lexsort((-s, n, r, diag))
    rd, dd, ed = r[o], diag[o], r[o] + n[o]
    inside = (dd[1:] == dd[:-1]) & (((rd[:-1] >= rd[1:]) & (ed[:-1] <= ed[1:])) |
                                    ((rd[1:] >= rd[:-1]) & (ed[1:] <= ed[:-1])))
    keep = o[np.concatenate([[True], ~inside])]
    keep = keep[np.lexsort((-s[keep], n[keep], r[keep], q[keep]))]
    out = np.zeros(a.size, dtype=SEGMENT_PAIR)
    out[:keep.size] = a[keep]
    return (torch.from_numpy(out.view(np.uint8).copy()),
            torch.tensor([keep.size], dtype=torch.int32))
