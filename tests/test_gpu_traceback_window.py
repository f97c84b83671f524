"""The traceback stage's DP with its band in registers, and where it gives way to
the one with rows in memory, against the oracle: query lengths around the 32
cells that the walk back takes at once, X-drops whose first row (X-drop - 10
columns at gap costs 11/1) just fits the 192 columns of registers and just does
not, alignments with long gaps, and direction buffers of odd and tiny sizes. Which
form a call takes first goes by the X-drop; both sides of that line are in
test_gpu_traceback_forms.py."""
import numpy as np
import pytest

from blaze103 import synth

from _parity import concat
from test_gpu_traceback import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qlen", [31, 32, 33, 64, 65, 513])
@pytest.mark.parametrize("xdrop,cap", [(12, 65536), (64, 65536), (64, 333), (202, 65536), (203, 65536), (400, 65)])
def test_traceback_window(qlen, xdrop, cap, monkeypatch):
    monkeypatch.setenv("BLAZE_INITIAL_TRACEBACK_CAP", str(cap))
    rng = np.random.default_rng(qlen + xdrop)
    q = synth.random_residues(rng, qlen)
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(1, 400, 40)]
    for gap in (1, 2, 31, 32, 33, 60, 100):
        cut = qlen // 2
        extra = synth.random_residues(rng, gap)
        seqs.append(np.concatenate([seqs[gap % 40], q[:cut], extra, q[cut:], seqs[1]]))
        if gap < cut - 12:
            seqs.append(np.concatenate([q[:cut], q[cut + gap:]]))
    seqs += [synth.mutate(rng, np.concatenate([q, q]), 0.8), q.copy(), q[3:], q[:-3]]
    res, off = concat(seqs)
    got = _check(q, res, off, final_xdrop=xdrop)
    assert len(got) >= 8
