"""Groups of which a warp stages only a part at a time, against the oracle: query
lengths on both sides of the one from which it does, and of a batch."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shortest", [1, 60])
def test_groups_staged_in_parts(shortest):
    rng = np.random.default_rng(31)
    qs = [synth.random_residues(rng, L) for L in (1300, 1301, 2600)]
    n = 60_000
    lengths = rng.integers(shortest, 400, n)
    seqs = np.split(synth.random_residues(rng, int(lengths.sum())), np.cumsum(lengths)[:-1])
    for i in rng.choice(n, 400, replace=False):
        q = qs[int(rng.integers(0, 3))]
        s0 = int(rng.integers(0, len(q) - 120))
        seqs[i] = np.concatenate([seqs[i], synth.mutate(rng, q[s0:s0 + 120], 0.7)])
    res, off = concat(seqs)
    assert len(res) > 2240 * 152 * 32
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(q), db.tot_len, db.num_seqs)[0] for q in qs]
    got = ps.run_batch(blaze103.QueryBatch(db, qs), params)
    for i, q in enumerate(qs):
        want, _, _ = compare(q, res, off, seq_src=db, search=ps)
        assert len(want) > 50
        for f in ("oid", "score", "q_start", "s_end"):
            assert np.array_equal(got[got["query"] == i][f], want[f])
    ps.close()
    db.close()
