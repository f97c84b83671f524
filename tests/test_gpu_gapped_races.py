"""The gapped stage where its warps read what others are writing, against the
oracle: subjects whose many init hits lie inside the HSP of their best one, so
that whether a DP is skipped depends on what has ended by then, and a flag that
is raised while other blocks start. The outcome may not."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat
from test_zz_no_alloc import MAX_INIT, MAX_SUBJECT, TOO_MANY_INIT, _assert_equal, _Caller, _groups, _regular, _workload

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


def test_flagged_items_leave_the_others():
    pytest.importorskip("torch")
    q, res, off = _workload()
    p, want, init = _regular(q, res, off)
    hits, groups = _groups(init)
    # the first subjects carry one init hit more than the entry point takes
    crowded = groups[:6]
    many = np.concatenate([np.repeat(hits[int(g["first"]):int(g["first"]) + 1], MAX_INIT + 1, axis=0) for g in crowded])
    bad = groups.copy()
    bad["n"][:6] = MAX_INIT + 1
    bad["first"][:6] = len(hits) + (MAX_INIT + 1) * np.arange(6)
    caller = _Caller(q, res, off, len(want) + 64)
    rest = want[~np.isin(want["oid"], crowded["subject"])]
    for call in range(20):
        st, got, flags = caller.call(np.concatenate([hits, many]), bad, MAX_SUBJECT, MAX_INIT, p)
        assert st == 0 and flags == TOO_MANY_INIT
        _assert_equal(got, rest, f"call {call}")
