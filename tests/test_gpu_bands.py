"""Scan launches in bands of diagonals, against the oracle: subjects cut in
pieces (lengths around a piece's), tables of one band at the query lengths
where the kinds of table change, both with HSPs that run along a band's edge
diagonals, tiny init-hit and scratch buffers, and long queries of a batch."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import compare, concat, params_for

pytestmark = pytest.mark.gpu


def _workload(rng, qlen, longest):
    q = synth.random_residues(rng, qlen)
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 300, 80)]
    for L in (0, 1, 112, 113, 114, 128, 240, 241, 242, 2224, 2225, 2226, longest):
        s = synth.random_residues(rng, L)
        for at in range(0, max(L - 150, 0), 400):  # matches on many diagonals
            w = min(qlen, 90)
            s0 = int(rng.integers(0, qlen - w + 1))
            m = synth.mutate(rng, q[s0:s0 + w], 0.75)[:L - at]
            s[at:at + len(m)] = m
        seqs.append(s)
    seqs.append(np.tile(synth.random_residues(rng, 3), 300))
    return q, *concat(seqs)


@pytest.mark.parametrize("qlen,longest", [(3, 9000), (60, 33_000), (1000, 33_000), (7000, 5000), (7001, 5000),
                                          (7001, 33_000), (11_777, 2500), (14_336, 2500), (14_337, 2500),
                                          (32_000, 6000)])
@pytest.mark.parametrize("window", [40, 256, 257])
def test_bands_against_the_oracle(qlen, longest, window):
    rng = np.random.default_rng(qlen + longest)
    q, res, off = _workload(rng, qlen, longest)
    got, _, _ = compare(q, res, off, window=window, ungapped_cutoff=25)
    assert qlen < 60 or len(got) >= 10


@pytest.mark.parametrize("qlen", [300, 7500])
def test_bands_with_tiny_buffers(qlen, monkeypatch):
    for name in ("SCRATCH", "INIT", "OUT", "WORK"):
        monkeypatch.setenv(f"BLAZE_INITIAL_{name}_CAP", "1")
    rng = np.random.default_rng(5)
    q, res, off = _workload(rng, qlen, 20_000)
    _, _, stats = compare(q, res, off, ungapped_cutoff=22)
    assert stats["reruns"] > 0


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_bands_in_a_batch(mode):
    rng = np.random.default_rng(6)
    qs = [synth.random_residues(rng, L) for L in (7100, 30, 12_000, 400, 15_000)]
    _, res, off = _workload(rng, 300, 12_000)
    db = blaze103.SeqSrc(res, off)
    ps = blaze103.PrelimSearch(db, autotune=False)
    ps.set_tuning(batch_launch=mode)
    params = [params_for(len(q), db.tot_len, db.num_seqs, ungapped_cutoff=20)[0] for q in qs]
    got = ps.run_batch(blaze103.QueryBatch(db, qs), params)
    assert len(got) > 0
    for i, q in enumerate(qs):
        want, _, _ = compare(q, res, off, seq_src=db, search=ps, ungapped_cutoff=20)
        mine = got[got["query"] == i]
        for f in ("oid", "score", "q_start", "q_end", "s_start", "s_end"):
            assert np.array_equal(mine[f], want[f])
    ps.close()
    db.close()
