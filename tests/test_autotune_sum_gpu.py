"""The contiguous autotuner: two names of one kernel are one candidate, and
what the choice is kept for: calls that write every
pair's count, not the sum alone (two launches, from the columns' counts; a pair
kernel takes one)."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _container(sb, n=300, m=5000):
    words = gen.bernoulli_rows(n, m, (0.05, 0.6), 903)
    c = sb.StormContig(m)
    c.add_bitmaps(words)
    return c, ol.contig_matrix(words)


def test_sum_after_autotune(sb):
    c, (want, ws) = _container(sb)
    assert c.pairw_intersect_cardinality() == ws and c.last_launches() == 2
    k, _, _ = c.autotune()
    assert c.pairw_intersect_cardinality() == ws and c.last_launches() == 2
    got, s = c.matrix()                                  # the tuned choice, one launch
    assert s == ws and c.last_kernel() == k and c.last_launches() == 1
    np.testing.assert_array_equal(got, want)
    c.set_kernel(sb.KERNEL_POPC)                         # a kernel asked for by name runs
    assert c.pairw_intersect_cardinality() == ws and c.last_launches() == 1
    assert c.last_kernel() == sb.KERNEL_POPC
    c.close()


def test_autotune_without_rows_keeps_the_choice(sb):
    c = sb.StormContig(5000)
    c.set_kernel(sb.KERNEL_MMA)
    assert c.autotune()[0] == sb.KERNEL_MMA
    words = gen.bernoulli_rows(40, 5000, (0.05, 0.6), 904)
    c.add_bitmaps(words)
    assert c.pairw_intersect_cardinality() == ol.contig_matrix(words)[1]
    assert c.last_launches() == 1 and c.last_kernel() == sb.KERNEL_MMA
    c.close()


@pytest.mark.parametrize("m", (5000, 65536))
def test_one_kernel_under_two_names_is_timed_once(sb, m):
    """MMA and MMA_DB share a kernel up to 2^24 bits: the same times, and a
    choice between the two that noise has no part in (the first)."""
    c, (want, ws) = _container(sb, 700, m)
    k, _, times = c.autotune()
    assert times[2] == times[0] > 0 and times[3] == times[1] > 0
    assert k != sb.KERNEL_MMA_DB
    assert c.matrix()[1] == ws
    c.close()
