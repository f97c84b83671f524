"""Which launch form a batched run takes by itself, told by the number of kernels:
one for the batch against few residues or with a long subject, one per query
otherwise; the results are the same in every form."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("residues,longest,one", [(300_000, 60, True), (8_000_000, 300, True), (8_500_000, 300, False),
                                                  (8_500_000, 9000, True)])
def test_automatic_form(residues, longest, one):
    rng = np.random.default_rng(longest)
    qs = [synth.random_residues(rng, int(L)) for L in rng.integers(20, 400, 12)]
    lengths = np.minimum(rng.integers(20, 300, residues // 40), min(longest, 300))
    lengths = lengths[:np.searchsorted(np.cumsum(lengths), residues)]
    seqs = np.split(synth.random_residues(rng, int(lengths.sum())), np.cumsum(lengths)[:-1])
    for i, q in enumerate(qs):
        seqs[i * 50] = synth.mutate(rng, q, 0.7)[:min(longest, 300)]
    seqs.append(synth.random_residues(rng, longest))
    res, off = concat(seqs)
    assert (len(res) < 2**23) == (residues < 2**23) and len(res) // (152 * 32) < 9000
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(q), db.tot_len, db.num_seqs)[0] for q in qs]
    batch = blaze103.QueryBatch(db, qs)
    outs, launches = [], []
    for mode in (0, 1, 2):
        ps.set_tuning(batch_launch=mode)
        outs.append(ps.run_batch(batch, params))
        launches.append(ps.stats()["kernel_launches"])
    assert launches[1] < len(qs) <= launches[2]
    assert launches[0] == launches[1 if one else 2]
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    for i in (0, 7):
        want, _, _ = compare(qs[i], res, off, seq_src=db, search=ps)
        mine = outs[0][outs[0]["query"] == i]
        for f in ("oid", "score", "q_start", "q_end", "s_start", "s_end"):
            assert np.array_equal(mine[f], want[f]), (i, f)
    batch.close()
    ps.close()
    db.close()


@pytest.mark.parametrize("subjects,longest,queries", [(1, 30, 300), (40, 20, 1000), (3000, 60, 90), (3000, 60, 400),
                                                      (800, 900, 400)])
def test_batches_against_small_databases(subjects, longest, queries):
    # groups cut for one query's pass and for a launch of many
    rng = np.random.default_rng(subjects + queries)
    qs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 80, queries)]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(0, longest + 1, subjects)]
    for i in range(0, subjects, 4):
        seqs[i] = np.concatenate([seqs[i], synth.mutate(rng, qs[i % queries], 0.8)])
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    over = dict(ungapped_cutoff=18, gapped_cutoff=18)
    params = [params_for(len(q), db.tot_len, db.num_seqs, **over)[0] for q in qs]
    batch = blaze103.QueryBatch(db, qs)
    outs = []
    for stage, mode in ((0, 0), (128, 1), (0, 2)):
        ps.set_tuning(batch_launch=mode, stage_bytes=stage)
        outs.append(ps.run_batch(batch, params))
        assert np.array_equal(outs[0], outs[-1])
    assert len(outs[0]) > 0
    for i in range(0, queries, 37):
        want, _, _ = compare(qs[i], res, off, seq_src=db, search=ps, **over)
        mine = outs[0][outs[0]["query"] == i]
        for f in ("oid", "score", "q_start", "q_end", "s_start", "s_end"):
            assert np.array_equal(mine[f], want[f]), (i, f)
    batch.close()
    ps.close()
    db.close()
