"""Timed cases of the BLASTP preliminary search and its traceback.

Each case is one program's use of the library against a database that stays
resident on the GPU: the one-call drop-in, a search object given one query, a
batch of queries, the serving loop, and the traceback after a search. The
databases are synthetic protein sequences of the shape the benchmark uses
(log-normal lengths, Robinson-Robinson composition, planted homologs,
low-complexity runs), made from the seed.

`listed` holds the fixed cases, `draw` one more of the same ranges, `prepare`
makes what a program has in hand before the call, `run` makes the call and
`work` says what the call cannot do without.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blaze-sc-ad_gb300"))

import blaze103  # noqa: E402
from blaze103 import synth  # noqa: E402

MEAN_LENGTH = 350.0  # of the synthetic subjects (median 250, sigma 0.82)
MUTANTS = 400        # distinct homologs planted in one database, at most


def _case(name, call, queries, qlen, subjects, *, qlen_to=0, max_len=5000, homologs=0.01, identity=0.40,
          low_complexity=0.0, evalue=10.0, hitlist=0):
    """queries of qlen residues, or spread geometrically over qlen..qlen_to."""
    return {"name": name, "call": call, "queries": queries, "qlen": qlen, "qlen_to": qlen_to, "subjects": subjects,
            "max_len": max_len, "homologs": homologs, "identity": identity, "low_complexity": low_complexity,
            "evalue": evalue, "hitlist": hitlist}


def listed():
    return [
        # a peptide against a handful of sequences: launches, copies and host work only
        _case("peptide vs 500", "one_call", 1, 31, 500, homologs=0.05),
        # one ordinary protein against a proteome-sized database, as a notebook calls it
        _case("protein vs proteome", "run", 1, 300, 20_000),
        # a short domain against a mid-sized database
        _case("domain vs 400k", "one_call", 1, 103, 400_000),
        # the drop-in's headline: eight queries one after another against 0.7 G residues
        _case("eight queries vs 2M", "one_call", 8, 100, 2_000_000, qlen_to=1000),
        # a multi-domain protein against long, repetitive subjects (titin-like lengths)
        _case("4,999 aa vs long subjects", "run", 1, 4999, 50_000, max_len=35_000, homologs=0.25, identity=0.45,
              low_complexity=0.20),
        # longer than the query copy in shared memory holds
        _case("12,345 aa vs proteome", "run", 1, 12_345, 20_000),
        # a few queries in one batch, the least a serving loop forms
        _case("batch of 5 vs 100k", "batch", 5, 120, 100_000, qlen_to=900, homologs=0.10),
        # a proteome's worth of queries in one batched call
        _case("batch of 256 vs 100k", "batch", 256, 50, 100_000, qlen_to=2000, homologs=0.10),
        # long queries in a batch, hit lists culled as max_target_seqs does
        _case("batch of 16 long", "batch", 16, 2000, 30_000, qlen_to=5000, max_len=35_000, homologs=0.25,
              identity=0.45, low_complexity=0.20, hitlist=500),
        # queries arriving at the serving loop
        _case("serve 64 vs 100k", "serve", 64, 30, 100_000, qlen_to=1500),
        # alignments of a finished search
        _case("traceback of a search", "traceback", 1, 500, 400_000),
        # search and alignments of a batch, hit lists culled, a strict expect value
        _case("batch of 32 with alignments", "batch_traceback", 32, 100, 30_000, qlen_to=1200, homologs=0.15,
              evalue=0.001, hitlist=100),
    ]


# word lookups of a drawn case at most: database residues x query residues
_DRAW_MOST = 1.2e12


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["one_call", "one_call", "run", "run", "batch", "batch", "serve", "traceback",
                       "batch_traceback"])
    many = call in ("batch", "serve", "batch_traceback")
    subjects = spread(300, 1_500_000 if not many else 300_000)
    qlen = spread(30, 12_500 if not many else 3000)
    qlen_to = spread(qlen, 5000) if many and qlen < 5000 else 0
    queries = spread(2, 300) if many else 1
    while queries > 1 and subjects * MEAN_LENGTH * queries * max(qlen, qlen_to) > _DRAW_MOST:
        queries = max(1, queries // 2)
    while subjects > 300 and subjects * MEAN_LENGTH * queries * max(qlen, qlen_to) > _DRAW_MOST:
        subjects = max(300, subjects // 2 + rng.randrange(7))
    c = _case("", call, queries, qlen, subjects, qlen_to=qlen_to, max_len=rng.choice([2000, 5000, 35_000]),
              homologs=round(rng.uniform(0.005, 0.20), 3), identity=round(rng.uniform(0.30, 0.60), 2),
              low_complexity=rng.choice([0.0, 0.0, 0.05, 0.20]), evalue=rng.choice([10.0, 10.0, 0.001]),
              hitlist=rng.choice([0, 0, 100, 500]) if call != "serve" else 0)
    del c["name"]
    return c


def _query_lengths(case):
    if case["queries"] == 1 or case["qlen_to"] <= case["qlen"]:
        return [case["qlen"]] * case["queries"]
    return [int(round(x)) for x in np.geomspace(case["qlen"], case["qlen_to"], case["queries"])]


def _plant(res, offsets, lengths, which, rows, row_len, rng):
    """Writes row i of `rows` (row_len[i] letters) into subject which[i], cut
    to its length, at a random place. `res` is on the GPU."""
    take = np.minimum(row_len, lengths[which])
    at = offsets[which] + (rng.random(len(which)) * (lengths[which] - take + 1)).astype(np.int64)
    take, at = torch.from_numpy(take).cuda(), torch.from_numpy(at).cuda()
    col = torch.arange(rows.shape[1], device="cuda")
    for lo in range(0, len(which), 1 << 16):  # in slices, so that the index tensors stay small
        m = col[None, :] < take[lo:lo + (1 << 16), None]
        pos = at[lo:lo + (1 << 16), None] + col[None, :]
        res[pos[m]] = rows[lo:lo + (1 << 16)][m]


def _database(case, queries, seed):
    """Residues and offsets: subjects in ascending length order."""
    rng = np.random.default_rng([seed, 1])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    n = case["subjects"]
    lengths = np.sort(synth.lognormal_lengths(rng, n, 250, 0.82, 30, min(case["max_len"], 5000)))
    n_long = n // 1000 if case["max_len"] > 5000 else 0
    if n_long:
        lengths[n - n_long:] = np.sort(rng.integers(15_000, case["max_len"] + 1, n_long))
    offsets = np.zeros(n + 1, np.int64)
    np.cumsum(lengths, out=offsets[1:])
    total = int(offsets[-1])
    letters = torch.from_numpy(synth.random_residues(rng, 1 << 16)).cuda()  # draws of the background composition
    res = torch.empty(total, dtype=torch.uint8, device="cuda")
    for lo in range(0, total, 1 << 26):
        hi = min(total, lo + (1 << 26))
        res[lo:hi] = letters[torch.randint(0, 1 << 16, (hi - lo,), device="cuda", dtype=torch.int32, generator=gen)]
    n_lc = int(case["low_complexity"] * n)
    if n_lc:  # runs of 50-200 residues over three letters
        which = rng.choice(n, n_lc, replace=False)
        abc = torch.from_numpy(rng.choice(synth.STD_CODES, (n_lc, 3))).cuda()
        pick = torch.randint(0, 3, (n_lc, 200), device="cuda", generator=gen)
        _plant(res, offsets, lengths, which, torch.gather(abc, 1, pick), rng.integers(50, 201, n_lc), rng)
    n_h = int(case["homologs"] * n)
    if n_h:
        pool = []
        for _ in range(min(n_h, MUTANTS)):
            q = queries[int(rng.integers(0, len(queries)))]
            w = int(min(rng.integers(100, 301), len(q)))
            s0 = int(rng.integers(0, len(q) - w + 1))
            pool.append(synth.mutate(rng, q[s0:s0 + w], case["identity"])[:400])
        table = np.zeros((len(pool), 400), np.uint8)
        for i, m in enumerate(pool):
            table[i, :len(m)] = m
        pool_len = np.array([len(m) for m in pool])
        which, row = rng.choice(n, n_h, replace=False), rng.integers(0, len(pool), n_h)
        _plant(res, offsets, lengths, which, torch.from_numpy(table).cuda()[torch.from_numpy(row).cuda()],
               pool_len[row], rng)
    return res.cpu().numpy(), offsets.astype(np.uint64)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 0])
    queries = [synth.random_residues(rng, L) for L in _query_lengths(case)]
    queries = [queries[i] for i in rng.permutation(len(queries))]
    db = blaze103.SeqSrc(*_database(case, queries, seed))
    params = []
    for q in queries:
        p = blaze103.default_params(len(q), db, case["evalue"])
        p.hitlist_size = case["hitlist"]
        params.append(p)
    s = {"call": case["call"], "rows": _rows(case), "queries": queries, "db": db, "params": params}
    if case["call"] == "serve":
        s["server"] = blaze103.Server(db, slots=3, max_batch=64, batch_window_us=200, evalue=case["evalue"])
        return s
    s["search"] = blaze103.PrelimSearch(db)
    if case["call"] in ("batch", "batch_traceback"):
        s["batch"] = blaze103.QueryBatch(db, queries)
    if case["call"] == "traceback":
        s["search"].run(queries[0], params[0])
    return s


def _rows(case):
    """HSPs of a pass at most: the size of the caller's result buffer."""
    per_query = 4 * case["hitlist"] if case["hitlist"] else case["subjects"]
    found = 3 * (case["homologs"] + case["low_complexity"]) * case["subjects"]
    return int(min(found, case["queries"] * per_query)) + 600 * case["queries"] + 500


def _fields(records, rows):
    """The records field by field in the caller's buffer of `rows` records
    (the rest of it stays zero)."""
    out = np.zeros(rows, records.dtype)
    out[:len(records)] = records
    return {f: out[f] for f in out.dtype.names if f not in ("reserved", "pad")}


def run(state):
    call, queries, params, rows = state["call"], state["queries"], state["params"], state["rows"]
    if call == "serve":
        server = state["server"]
        tickets = [server.submit(q) for q in queries]
        lists = [server.wait(t) for t in tickets]
        return {"hsps": _fields(np.concatenate(lists), rows), "count": np.array([len(x) for x in lists])}
    search = state["search"]
    if call == "one_call":
        lists = [search.prelim_search(q, p, rows) for q, p in zip(queries, params)]
        return {"hsps": _fields(np.concatenate(lists), rows), "count": np.array([len(x) for x in lists])}
    if call == "run":
        return {"hsps": _fields(search.run(queries[0], params[0]).hsps, rows)}
    if call == "traceback":
        return {"aligned": _fields(search.traceback(queries[0], params[0]), rows)}
    hsps = search.run_batch(state["batch"], params)
    if call == "batch":
        return {"hsps": _fields(hsps, rows)}
    aligned = search.traceback_batch(state["batch"], params)
    return {"hsps": _fields(hsps, rows), "aligned": _fields(aligned, rows)}


def work(case):
    """Bytes: the database (once per call; the one-call path is called once
    per query), the queries, the results. Operations: one word lookup per
    residue and query and one two-hit test per word hit (about one in 490
    pairs of a residue and a query residue), and the cells of the alignments."""
    residues = case["subjects"] * MEAN_LENGTH
    lengths = _query_lengths(case)
    kept = case["homologs"] * case["subjects"]  # subjects with an alignment, about
    if case["hitlist"]:
        kept = min(kept, case["hitlist"] * case["queries"])
    if case["call"] == "traceback":
        return {"bytes": kept * (500 + 72), "flops": kept * 17_000.0}
    calls = case["queries"] if case["call"] == "one_call" else 1
    ops = sum(residues * (1 + L / 490.0) for L in lengths)
    aligned = 17_000.0 * kept if case["call"] == "batch_traceback" else 0.0
    return {"bytes": calls * (residues + 8.0 * case["subjects"]) + sum(lengths) + 40.0 * kept, "flops": ops + aligned}
