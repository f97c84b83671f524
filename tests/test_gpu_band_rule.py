"""Searches on both sides of the line from which a query's launch runs in bands,
against the oracle: the longest subject one residue short of it and at it, in a
database whose shares are nothing beside it and in one where they count."""
import numpy as np
import pytest

from blaze103 import synth

from _parity import compare, concat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qlen", [4, 40, 400, 3920])
@pytest.mark.parametrize("others", [20, 9000])
@pytest.mark.parametrize("over", [-1, 0])
def test_both_sides_of_the_line(qlen, others, over):
    rng = np.random.default_rng(qlen + others)
    q = synth.random_residues(rng, qlen)
    seqs = [synth.random_residues(rng, int(L)) for L in rng.integers(30, 350, others)]
    total = sum(map(len, seqs))
    longest = -(-240_000 // (qlen + 80)) + (total // (152 * 32)) * 5 // 2 + over
    seqs.append(synth.random_residues(rng, longest))
    for i in list(range(0, others, 7)) + [others]:
        w = min(qlen, 80)
        s0 = int(rng.integers(0, qlen - w + 1))
        hom = synth.mutate(rng, q[s0:s0 + w], 0.75)[:len(seqs[i])]
        seqs[i][len(seqs[i]) - len(hom):] = hom
    res, off = concat(seqs)
    got, _, _ = compare(q, res, off, ungapped_cutoff=25, gapped_cutoff=25)
    assert qlen < 40 or len(got) >= 2
