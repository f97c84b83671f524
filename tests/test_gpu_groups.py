"""The word finder's groups of subjects and its two kinds of diagonal table,
against the oracle: subject lengths at the edges of the staging blocks and of
the scanned chunks, groups of the most subjects, subjects long enough that a
16-bit table has to be moved down, windows on both sides of the 16-bit limit
(query lengths at it: test_gpu_table_limits.py), queries in bands, and the batched
launch chosen by the longest subject."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat, params_for

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 3, 4, 13, 14, 15, 16, 17, 31, 32, 33, 110, 125, 126, 127, 128, 129, 130, 131, 255, 258]


def _subjects(rng, q, lengths, planted):
    seqs = [synth.random_residues(rng, int(L)) for L in lengths]
    for i in rng.choice(len(seqs), planted, replace=False):
        w = min(len(q), int(rng.integers(20, 120)))
        s0 = int(rng.integers(0, len(q) - w + 1))
        seqs[i] = np.concatenate([seqs[i], synth.mutate(rng, q[s0:s0 + w], 0.7)])
    return seqs


def test_groups_of_many_subjects():
    # 14 M residues in 31-subject groups and, for the longer ones, groups of a few
    rng = np.random.default_rng(71)
    q = synth.random_residues(rng, 300)
    lengths = rng.choice(EDGES, 200_000)
    res, off = concat(_subjects(rng, q, lengths, 3000))
    got, _, _ = compare(q, res, off, ungapped_cutoff=25)
    assert len(got) > 1000


@pytest.mark.parametrize("qlen,window", [(3, 40), (300, 256), (300, 257), (8192, 40), (8193, 40), (500, 2000)])
@pytest.mark.parametrize("stage_bytes", [0, 128, 16384])
def test_long_subjects_and_tables(qlen, window, stage_bytes):
    rng = np.random.default_rng(72)
    q = synth.random_residues(rng, qlen)
    run = np.tile(synth.random_residues(rng, 3), 400)  # every word hits itself along a whole diagonal band
    seqs = [synth.random_residues(rng, L) for L in EDGES + [16_300, 16_383, 33_000]]
    if qlen >= 100:
        seqs[-1][20_000:20_100] = q[:100]
        seqs[-2][:100] = q[-100:]
        seqs[-3][8000:9200] = run
        q[50:98] = run[:48]
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    ps.set_tuning(stage_bytes=stage_bytes)
    compare(q, res, off, seq_src=db, search=ps, window=window)
    ps.close()
    db.close()


@pytest.mark.parametrize("longest", [300, 30_000])
def test_batched_launch_by_longest_subject(longest):
    rng = np.random.default_rng(73)
    qs = [synth.random_residues(rng, L) for L in (4, 90, 300, 301, 1400, 9000)]
    seqs = _subjects(rng, qs[2], [int(x) for x in rng.integers(20, 290, 6000)], 300)
    seqs = [s[:longest] for s in seqs] + [synth.random_residues(rng, longest)]
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(q), db.tot_len, db.num_seqs)[0] for q in qs]
    batch = blaze103.QueryBatch(db, qs)
    outs = []
    for mode in (0, 1, 2):
        ps.set_tuning(batch_launch=mode, max_warps_per_block=4 if mode == 1 else 0)
        outs.append(ps.run_batch(batch, params))
    assert len(outs[0]) > 50
    for o in outs[1:]:
        assert np.array_equal(outs[0], o)
    for i, q in enumerate(qs):
        want, _, _ = compare(q, res, off, seq_src=db, search=ps)
        mine = outs[0][outs[0]["query"] == i]
        for f in ("oid", "score", "q_start", "q_end", "s_start", "s_end"):
            assert np.array_equal(mine[f], want[f]), (i, f)
    batch.close()
    ps.close()
    db.close()
