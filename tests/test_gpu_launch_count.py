"""The kernels that a run's statistics count: those of the one-call search include
the three that build the query's word lookup."""
import numpy as np
import pytest

import blaze103
from blaze103 import synth

from _parity import concat

pytestmark = pytest.mark.gpu


def test_one_call_counts_its_lookup():
    rng = np.random.default_rng(5)
    q = synth.random_residues(rng, 200)
    db = blaze103.SeqSrc(*concat([synth.random_residues(rng, 100), synth.mutate(rng, q, 0.7)]))
    ps = blaze103.PrelimSearch(db, autotune=False)
    p = blaze103.default_params(len(q), db)
    query = blaze103.Query(db, q)
    ps.run_query(query, p)
    resident = ps.stats()["kernel_launches"]
    ps.prelim_search(q, p, 64)
    assert ps.stats()["kernel_launches"] == resident + 3
    query.close()
    ps.close()
    db.close()
