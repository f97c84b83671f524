"""The order of the HSP lists, by query and then OID, for numbers of lists
around the one from which they are sorted by digits and subject numbers of
several digits, against the oracle."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import HSP_FIELDS, compare, concat, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_subjects", [3000, 70_000])
@pytest.mark.parametrize("lists", [1, 255, 256, 257, 2900])
def test_lists_by_query_and_oid(lists, n_subjects):
    rng = np.random.default_rng(lists)
    qs = [synth.random_residues(rng, 40 + 10 * i) for i in range(3)]
    seqs = [np.full(1, 1, np.uint8)] * n_subjects
    for i in rng.choice(n_subjects, lists, replace=False):
        seqs[i] = qs[int(rng.integers(0, 3))] if lists > 2000 else np.concatenate(qs)
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(q), db.tot_len, db.num_seqs)[0] for q in qs]
    batch = blaze103.QueryBatch(db, qs)
    got = ps.run_batch(batch, params)
    for i, q in enumerate(qs):
        want, _, stats = compare(q, res, off, seq_src=db, search=ps)
        assert lists > 2000 or stats["subjects_with_hsps"] == lists
        mine = got[got["query"] == i]
        for f in ["oid", "evalue"] + HSP_FIELDS:
            assert np.array_equal(mine[f], want[f])
    assert np.all(np.diff(got["query"].astype(np.int64)) >= 0)
    ps.close()
    db.close()
