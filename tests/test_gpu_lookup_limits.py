"""The word lookup at its limits, against the oracle: queries with more list entries
than 24 bits number (the packed cells cannot hold where the later words' lists
begin), and thresholds low enough for words with the letter 0."""
import numpy as np
import pytest

import blaze103
import oracle
from blaze103 import synth

from _parity import HSP_FIELDS, compare, concat, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qlen,threshold,fits", [(4700, 0, True), (4900, 0, False), (9000, 1, False),
                                                 (15_000, 0, False), (32_000, 4, False)])
def test_lists_beyond_24_bits(qlen, threshold, fits):
    rng = np.random.default_rng(17)
    q = synth.random_residues(rng, qlen)
    assert (len(oracle.lookup(q, threshold)[1]) < 2**24) == fits
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 60, 30)]
    for at in (0, qlen // 2, qlen - 60):  # words from the whole alphabet, so lists from the whole array
        seqs.append(synth.mutate(rng, q[at:at + 60], 0.8))
    seqs.append(np.arange(1, 28, dtype=np.uint8)[::-1].copy())
    res, off = concat(seqs)
    over = dict(word_threshold=threshold, ungapped_cutoff=30)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    want, _, _ = compare(q, res, off, seq_src=db, search=ps, **over)
    assert len(want) >= 3
    p, _ = params_for(qlen, db.tot_len, db.num_seqs, **over)
    one = ps.prelim_search(q, p, 65536)
    batch = blaze103.QueryBatch(db, [q[:200], q], threshold)
    got = ps.run_batch(batch, [params_for(200, db.tot_len, db.num_seqs, **over)[0], p])
    batch.close()
    got = got[got["query"] == 1]
    for f in ["oid"] + HSP_FIELDS:
        assert np.array_equal(one[f], want[f])
        assert np.array_equal(got[f], want[f])
    ps.close()
    db.close()


# a word with one letter 0 scores -32,746 at most; no residue is 0
@pytest.mark.parametrize("threshold", [-32_745, -32_746, -40_000, -100_000, -(2**31), 2**31 - 1])
@pytest.mark.parametrize("stage_bytes", [0, 128])
def test_thresholds_that_the_letter_0_reaches(threshold, stage_bytes):
    rng = np.random.default_rng(23)
    qs = [synth.random_residues(rng, L) for L in (2, 12, 300)]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(0, 90, 50)]
    seqs += [np.concatenate([synth.random_residues(rng, 9), q[:60]]) for q in qs] + [synth.random_residues(rng, 3000)]
    res, off = concat(seqs)
    over = dict(word_threshold=threshold, ungapped_cutoff=12)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    ps.set_tuning(stage_bytes=stage_bytes)
    batch = blaze103.QueryBatch(db, qs, threshold)
    got = ps.run_batch(batch, [params_for(len(q), db.tot_len, db.num_seqs, **over)[0] for q in qs])
    batch.close()
    for i, q in enumerate(qs):
        want, _, _ = compare(q, res, off, seq_src=db, search=ps, **over)
        for f in ["oid"] + HSP_FIELDS:
            assert np.array_equal(got[got["query"] == i][f], want[f])
    ps.close()
    db.close()
