"""Host rows that go to their places by copies with two pitches (640 words and
more, as shorter ones do when there is no memory to stage them): ragged lengths,
repeated calls on one container, few rows and several panels."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", (639, 640, 641, 1023, 1024))
def test_matrix_from_host_long_rows(sb, words):
    m = 64 * words - 7
    c = sb.StormContig(m)
    for n, seed in ((1100, 81), (3, 82), (300, 83)):
        rows = gen.bernoulli_rows(n, m, (0.05, 0.5), seed)
        want, ws = ol.contig_matrix(rows)
        got, s = c.matrix_from_host(rows)
        assert s == ws and len(c) == n
        np.testing.assert_array_equal(got, want, err_msg=str(n))
    c.close()
