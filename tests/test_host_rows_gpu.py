"""The ways host rows take to their places: one copy where they lie a pitch apart,
copies with two pitches (640 words and more, as shorter ones when there is no
memory to stage them; multiples of 512 words), and staged ones; ragged lengths,
repeated calls on one container, few rows and several panels."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", (1, 7, 8, 9, 64, 312, 313, 512, 639, 640, 641, 1023, 1024))
def test_matrix_from_host_row_lengths(sb, words):
    m = 64 * words - 7
    c = sb.StormContig(m)
    for n, seed in ((1100, 81), (3, 82), (300, 83)):
        rows = gen.bernoulli_rows(n, m, (0.05, 0.5), seed)
        want, ws = ol.contig_matrix(rows)
        got, s = c.matrix_from_host(rows)
        assert s == ws and len(c) == n
        np.testing.assert_array_equal(got, want, err_msg=str(n))
    c.close()
