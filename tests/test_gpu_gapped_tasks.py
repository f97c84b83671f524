"""The gapped stage's DP tasks against the oracle: one warp per DP with its band
in the register window (one half, both, moved on, outgrown), and one lane per DP,
which a batch takes only when it holds very many init hits (the limit is lowered
here)."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat, params_for

pytestmark = pytest.mark.gpu

FIELDS = ("oid", "score", "q_start", "q_end", "s_start", "s_end", "q_gapped_start", "s_gapped_start")


def _workload(seed=81, n=800, qlen=420):
    rng = np.random.default_rng(seed)
    q = synth.random_residues(rng, qlen)
    seqs = [synth.random_residues(rng, int(L)) for L in synth.lognormal_lengths(rng, n, 150, 0.8, 1, 3000)]
    for i in range(0, n, 3):  # related by 40-95 %, with insertions up to wider than the window
        w = int(rng.integers(20, qlen + 1))
        s0 = int(rng.integers(0, qlen - w + 1))
        hom = synth.mutate(rng, q[s0:s0 + w], float(rng.uniform(0.4, 0.95)), indel_rate=0.04)
        if i % 9 == 0:
            k = int(rng.integers(0, len(hom) + 1))
            hom = np.concatenate([hom[:k], synth.random_residues(rng, int(rng.integers(20, 90))), hom[k:]])
        seqs[i] = np.concatenate([seqs[i][:40], hom, seqs[i][40:]])
    return q, concat(seqs)


@pytest.mark.parametrize("xdrop,gap_open,gap_extend", [(12, 11, 1), (38, 11, 1), (75, 11, 1), (130, 11, 1),
                                                       (400, 11, 1), (60, 5, 3), (90, 40, 1), (38, 0, 2)])
def test_register_window(xdrop, gap_open, gap_extend):
    q, (res, off) = _workload()
    got, _, stats = compare(q, res, off, gapped_xdrop=xdrop, gap_open=gap_open, gap_extend=gap_extend)
    assert len(got) > 100 and stats["gapped_extensions"] > 100


@pytest.mark.parametrize("qlen", [3, 31, 33, 64, 129])
def test_short_queries(qlen):
    q, (res, off) = _workload(82 + qlen, 300, max(qlen, 20))
    compare(q[:qlen], res, off, ungapped_cutoff=15, gapped_cutoff=15)


@pytest.mark.parametrize("slots", ["0", "400"])
@pytest.mark.parametrize("override", [{}, {"gapped_xdrop": 100}, {"gap_open": 40}])
def test_lane_per_dp(monkeypatch, slots, override):
    monkeypatch.setenv("BLAZE_LANE_DP_SLOTS", slots)
    monkeypatch.setenv("BLAZE_INITIAL_INIT_CAP", "64")
    q, (res, off) = _workload()
    rng = np.random.default_rng(83)
    qs = [q] + [synth.random_residues(rng, int(L)) for L in rng.integers(10, 900, 18)]
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    params = [params_for(len(x), db.tot_len, db.num_seqs, **override)[0] for x in qs]
    batch = blaze103.QueryBatch(db, qs)
    out = ps.run_batch(batch, params)
    want, _, _ = compare(q, res, off, seq_src=db, search=ps, **override)
    mine = out[out["query"] == 0]
    assert len(mine) == len(want) > 100
    for f in FIELDS:
        assert np.array_equal(mine[f], want[f]), f
    batch.close()
    ps.close()
    db.close()
