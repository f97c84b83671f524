"""The word lookup built on the device, against the oracle: query lengths around
a word and around the parts of 256 offsets, the longest query, thresholds from "nearly
every word" (cells of more than 255 offsets) to "the exact word only", in the
plain, one-call and batched forms."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import HSP_FIELDS, compare, concat, params_for

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 257, 258, 259, 511, 512, 513, 514, 515, 1026, 1027]


@pytest.mark.parametrize("qlens,threshold", [(LENGTHS, 11), (LENGTHS, 40), ([32_000], 11), ([300, 2000], 0),
                                             ([300, 2000], 4)])
def test_lookup_against_the_oracle(qlens, threshold):
    rng = np.random.default_rng(91)
    qs = [synth.random_residues(rng, L) for L in qlens]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 200, 60)]
    for i, q in enumerate(qs):
        w = min(len(q), 80)
        seqs.append(synth.mutate(rng, q[len(q) - w:], 0.8))
    seqs.append(np.arange(1, 28, dtype=np.uint8))
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(q), db.tot_len, db.num_seqs, word_threshold=threshold, ungapped_cutoff=20)[0] for q in qs]
    batch = blaze103.QueryBatch(db, qs, threshold)
    got = ps.run_batch(batch, params)
    batch.close()
    for i, q in enumerate(qs):
        want, _, _ = compare(q, res, off, seq_src=db, search=ps, word_threshold=threshold, ungapped_cutoff=20)
        one = ps.prelim_search(q, params[i], 4096)
        mine = got[got["query"] == i]
        for f in ["oid"] + HSP_FIELDS:
            assert np.array_equal(one[f], want[f])
            assert np.array_equal(mine[f], want[f])
    ps.close()
    db.close()
