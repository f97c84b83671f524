"""The largest diagonal tables, against the oracle: query and window lengths up to
the most that shared memory holds, in the plain and both batched forms, and the
16-bit table at its longest query, with subjects long enough that it has to be
moved down and a match along nearly the whole query."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import HSP_FIELDS, compare, concat, params_for

pytestmark = pytest.mark.gpu


def _batched(db, ps, qs, mode, want, **over):
    ps.set_tuning(batch_launch=mode)
    batch = blaze103.QueryBatch(db, qs)
    got = ps.run_batch(batch, [params_for(len(q), db.tot_len, db.num_seqs, **over)[0] for q in qs])
    batch.close()
    for i, w in enumerate(want):
        mine = got[got["query"] == i]
        for f in ["oid"] + HSP_FIELDS:
            assert np.array_equal(mine[f], w[f]), (mode, i, f)


# 55,888 residues: the most with the presence bitset, 56,432: what the same
# tuning took before subjects were grouped, 56,688: the most without the bitset
@pytest.mark.parametrize("qlen,window", [(32_000, 23_888), (32_000, 23_889), (32_000, 24_432), (8193, 48_239),
                                         (100, 56_304), (32_000, 24_688), (100, 56_588)])
def test_longest_tables(qlen, window):
    rng = np.random.default_rng(qlen)
    qs = [synth.random_residues(rng, qlen), synth.random_residues(rng, min(qlen, 700))]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(0, 400, 60)] + [synth.random_residues(rng, 9000)]
    for q in qs:
        for at in (0, len(q) - 90):
            seqs.append(np.concatenate([synth.random_residues(rng, 40), synth.mutate(rng, q[at:at + 90], 0.7)]))
        seqs[60][1000:1060] = q[20:80]
    seqs.append(np.tile(synth.random_residues(rng, 3), 300))
    res, off = concat(seqs)
    over = dict(window=window, ungapped_cutoff=30)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    want = [compare(q, res, off, seq_src=db, search=ps, **over)[1] for q in qs]
    assert min(len(w) for w in want) >= 2
    want = [dict(oid=w["subject"], **{f: w[f] for f in HSP_FIELDS}) for w in want]
    for mode in (1, 2):
        _batched(db, ps, qs, mode, want, **over)
    ps.close()
    db.close()


def test_beyond_the_longest_table():
    rng = np.random.default_rng(3)
    q = synth.random_residues(rng, 32_000)
    db = blaze103.SeqSrc(*concat([q[:200]]))
    ps = blaze103.PrelimSearch(db, autotune=False)
    p, _ = params_for(len(q), db.tot_len, 1, window=24_689)
    with pytest.raises(blaze103.BlazeError):
        ps.run(q, p)
    ps.close()
    db.close()


@pytest.mark.parametrize("qlen", [11_776, 11_777])
def test_longest_16_bit_table(qlen):
    rng = np.random.default_rng(qlen)
    q = synth.random_residues(rng, qlen)
    seqs = [synth.random_residues(rng, int(L)) for L in (1, 300, 2240, 16_383, 16_384, 33_000)]
    seqs[4][3000:3000 + qlen - 60] = q[30:qlen - 30]  # along a diagonal, within a moved table
    seqs[5][20_000:20_000 + qlen] = q
    seqs.append(q.copy())
    seqs.append(np.concatenate([q[5000:], q[:5000]]))
    res, off = concat(seqs)
    over = dict(window=256)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    want, _, _ = compare(q, res, off, seq_src=db, search=ps, **over)
    assert len(want) >= 4
    for mode in (1, 2):
        _batched(db, ps, [q], mode, [want], **over)
    ps.close()
    db.close()
