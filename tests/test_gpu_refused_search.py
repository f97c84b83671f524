"""One-call searches right after one that is refused, against the oracle: the
refused call's residues are staged and its lookup is started before the refusal."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import HSP_FIELDS, concat, oracle_run, params_for

pytestmark = pytest.mark.gpu


def test_search_after_a_refused_one():
    rng = np.random.default_rng(41)
    long_q = synth.random_residues(rng, 32_000)
    qs = [synth.random_residues(rng, int(L)) for L in (32_000, 40, 900, 31_990, 5, 2000)]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 300, 80)]
    for q in qs:
        seqs.append(synth.mutate(rng, q[-min(len(q), 90):], 0.8))
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    refused, _ = params_for(len(long_q), db.tot_len, db.num_seqs, window=60_000)
    for q in qs * 3:
        p, pd = params_for(len(q), db.tot_len, db.num_seqs, ungapped_cutoff=25)
        with pytest.raises(blaze103.BlazeError):
            ps.prelim_search(long_q, refused, 16)
        got = ps.prelim_search(q, p, 65536)
        want, _ = oracle_run(q, res, off, pd)
        assert np.array_equal(got["oid"], want["subject"])
        for f in HSP_FIELDS:
            assert np.array_equal(got[f], want[f])
    ps.close()
    db.close()
