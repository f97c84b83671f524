"""Gap costs and X-drops far above the usual ones against the oracle: an X-drop
that never ends a DP, gap costs that forbid gaps, both near the 32 bits that the
DPs compute in. Sequences are short, so that every band fits the registers."""
import numpy as np
import pytest

import blaze103
import oracle
from blaze103 import synth

from _parity import compare, concat, params_for
from test_gpu_traceback import TB_FIELDS

pytestmark = pytest.mark.gpu

MOST = 2**31 - 1


@pytest.mark.parametrize("gap_open,gap_extend,xdrop", [(11, 1, MOST), (11, 1, 2**30 + 100), (32767, 1, MOST),
                                                       (11, 1, 2**29 - 400), (32767, 32767, 38), (0, 2**22, 38),
                                                       (11, 2**23, 400), (11, 2**24, 38), (2**28, 1, 38),
                                                       (2**20, 2**20, 2**29)])
def test_large_gap_costs_and_xdrops(gap_open, gap_extend, xdrop):
    rng = np.random.default_rng(7)
    q = synth.random_residues(rng, 45)
    seqs = []
    for _ in range(250):
        s0 = int(rng.integers(0, 15))
        s = synth.mutate(rng, q[s0:s0 + int(rng.integers(20, 45))], float(rng.uniform(0.6, 1.0)), indel_rate=0.03)
        seqs.append(np.concatenate([synth.random_residues(rng, int(rng.integers(0, 8))), s])[:52])
    res, off = concat(seqs)
    over = dict(gap_open=gap_open, gap_extend=gap_extend, gapped_xdrop=xdrop, ungapped_cutoff=14, gapped_cutoff=14,
                prelim_evalue=1e9)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db)
    try:
        _, want, _ = compare(q, res, off, seq_src=db, search=ps, **over)
        assert len(want) > 100
        p, pd = params_for(len(q), int(off[-1]), len(seqs), **over)
        got = ps.traceback(q, p, evalue=1e9, final_xdrop=xdrop)
    finally:
        ps.close()
        db.close()
    ref = oracle.traceback_hsps(q, res, off, want, pd, xdrop=xdrop, evalue=1e9)
    assert got["oid"].tolist() == [r["subject"] for r in ref]
    for f in TB_FIELDS:
        assert got[f].tolist() == [r[f] for r in ref], f
