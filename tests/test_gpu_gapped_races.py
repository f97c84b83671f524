"""The gapped stage where its warps read what others are writing, against the
oracle: subjects whose many init hits lie inside the HSP of their best one, so
that whether a DP is skipped depends on what has ended by then. The outcome may
not."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subjects", [1, 7, 700])
def test_skipped_dps(subjects):
    rng = np.random.default_rng(61)
    q = synth.random_residues(rng, 900)
    seqs = []
    for _ in range(subjects):
        m = synth.mutate(rng, q, float(rng.uniform(0.5, 0.9)), indel_rate=0.02)
        seqs.append(np.concatenate([synth.random_residues(rng, 10), m]))
    res, off = concat(seqs)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    first = None
    for _ in range(5):
        got, _, stats = compare(q, res, off, seq_src=db, search=ps, ungapped_cutoff=14, gapped_cutoff=14)
        counted = (len(got), stats["init_hsps"], stats["gapped_extensions"], stats["dp_cells"])
        first = first or counted
        assert counted == first
    ps.close()
    db.close()
