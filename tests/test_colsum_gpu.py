"""The sum over all pairs of dense rows from the columns' counts
(csrc/colsum.cuh), at the edges of its groups of eight rows, its 2048-column
blocks and its 2^22-column strips; whole numbers, equal to the oracle's."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", ((1, 1), (2, 64), (7, 2047), (8, 2048), (9, 2049), (65, 511), (600, 4097), (5000, 70),
                                 (40000, 64), (3, (1 << 22) + 65)))
def test_sum_matches_oracle(sb, n, m):
    words = gen.bernoulli_rows(n, m, (0.0, 1.0), n + m)
    cols = np.unpackbits(words.view(np.uint8), axis=1, bitorder="little").sum(axis=0, dtype=np.int64)
    want = int((cols * (cols - 1) // 2).sum())
    if n <= 600:
        assert want == ol.contig_matrix(words, want_matrix=False)[1]
    c = sb.StormContig(m)
    c.add_bitmaps(words)
    assert c.pairw_intersect_cardinality() == want
    assert c.pairw_intersect_cardinality(blocked=8) == want
    c.set_kernel(sb.KERNEL_MMA)
    assert c.pairw_intersect_cardinality() == want
