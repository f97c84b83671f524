"""A server's tuning of which only batch_launch is set reaches its searches: an
invalid value fails the queries as it does next to other fields, the valid ones
return the plain runs' results."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import concat

pytestmark = pytest.mark.gpu


def test_batch_launch_alone():
    rng = np.random.default_rng(51)
    qs = [synth.random_residues(rng, L) for L in (30, 300, 1500)]
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(20, 300, 300)]
    seqs += [synth.mutate(rng, q, 0.7) for q in qs] + [synth.random_residues(rng, 9000)]
    db = blaze103.SeqSrc(*concat(seqs))
    ps = blaze103.PrelimSearch(db, autotune=False)
    want = [ps.run(q).hsps for q in qs]
    ps.close()
    for mode in (1, 2):
        srv = blaze103.Server(db, slots=1, tuning=dict(batch_launch=mode))
        tickets = [srv.submit(q) for q in qs]
        for t, w in zip(tickets, want):
            got = srv.wait(t, 60_000)
            for f in blaze103.HSP_DTYPE.names:
                assert np.array_equal(got[f], w[f])
        srv.close()
    for tuning in (dict(batch_launch=3), dict(batch_launch=3, launch_mode=1)):
        srv = blaze103.Server(db, slots=1, tuning=tuning)
        with pytest.raises(blaze103.BlazeError) as e:
            srv.wait(srv.submit(qs[0]), 60_000)
        assert e.value.status == 1  # BLAZE_ERR_INVALID_ARG, as blaze_search_set_tuning
        srv.close()
    db.close()
