"""The traceback stage's two forms, bands in registers and rows in memory, against
the oracle: X-drops on both sides of the line between them at several gap costs,
databases whose subjects all fit the registers, gaps that make bands outgrow them
all the same, and direction buffers of odd and tiny sizes."""
import numpy as np
import pytest

import blaze103
import oracle
from blaze103 import synth

from _parity import concat, oracle_run, params_for
from test_gpu_traceback import TB_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [191, 192, 900])
@pytest.mark.parametrize("gap_open,gap_extend,xdrops", [(11, 1, (20, 64, 70, 71, 130, 300)), (5, 3, (64, 184, 185, 500)),
                                                        (60, 1, (119, 120, 400)), (0, 2, (38, 118, 120))])
@pytest.mark.parametrize("cap", [65536, 100])
def test_both_forms(longest, gap_open, gap_extend, xdrops, cap, monkeypatch):
    monkeypatch.setenv("BLAZE_INITIAL_TRACEBACK_CAP", str(cap))
    rng = np.random.default_rng(longest + gap_open)
    q = synth.random_residues(rng, 400)
    seqs = []
    for k in range(60):
        w = int(rng.integers(30, 400))
        s0 = int(rng.integers(0, 400 - w + 1))
        s = synth.mutate(rng, q[s0:s0 + w], float(rng.uniform(0.5, 0.95)), indel_rate=0.03)
        if k % 3 == 0:  # a long insertion
            at = int(rng.integers(0, len(s) + 1))
            s = np.concatenate([s[:at], synth.random_residues(rng, int(rng.integers(20, 120))), s[at:]])
        seqs.append(np.concatenate([s, synth.random_residues(rng, int(rng.integers(0, 300)))])[:longest])
    seqs.append(np.concatenate([q, q, q])[:longest])
    res, off = concat(seqs)
    p, pd = params_for(len(q), int(off[-1]), len(seqs), gap_open=gap_open, gap_extend=gap_extend, prelim_evalue=1e6)
    db = blaze103.SeqSrc(res, off)
    assert max(map(len, seqs)) == longest
    ps = blaze103.PrelimSearch(db)
    prelim, _ = oracle_run(q, res, off, pd)
    for xdrop in xdrops:
        assert len(ps.run(q, p).hsps) == len(prelim) > 30
        got = ps.traceback(q, p, evalue=1e6, final_xdrop=xdrop)
        ref = oracle.traceback_hsps(q, res, off, prelim, pd, xdrop=xdrop, evalue=1e6)
        assert got["oid"].tolist() == [r["subject"] for r in ref]
        for f in TB_FIELDS:
            assert got[f].tolist() == [r[f] for r in ref], (xdrop, f)
    ps.close()
    db.close()
