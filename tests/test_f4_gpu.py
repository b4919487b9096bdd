"""The 4-bit tensor-core kernel (csrc/bb_f4.cuh) at the edges of its tiles,
stages and counts: 256-row tiles, 512-bit stages, counts that no longer fit 16
bits (rows past 65535 bits), counts up to 2^24, and the first row length that
is left to the 8-bit kernels.  Whole numbers: every result equals the oracle's."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", (1, 511, 513, 1025, 65535, 65536, 66049))
@pytest.mark.parametrize("n", (1, 255, 257, 513))
def test_tile_and_stage_edges(sb, n, m):
    words = gen.bernoulli_rows(n, m, (0.3, 1.0), 31 * n + m)
    words[n // 2] = gen.bernoulli_rows(1, m, 1.1, 1)[0]          # one full row: the largest count
    want, ws = ol.contig_matrix(words)
    for kernel in (sb.KERNEL_MMA, sb.KERNEL_MMA_DB):
        for sched in (sb.SCHED_TILES, sb.SCHED_STREAM_K):
            c = sb.StormContig(m)
            c.set_kernel(kernel)
            c.set_schedule(sched)
            c.add_bitmaps(words)
            got, s = c.matrix()
            np.testing.assert_array_equal(got, want, err_msg=f"{kernel} {sched}")
            assert s == ws
            c.close()


@pytest.mark.parametrize("m", ((1 << 24) - 1, 1 << 24, (1 << 24) + 1))
def test_counts_up_to_the_accumulator_limit(sb, m):
    """Full rows with a few bits cleared one by one: counts m, m - 1, ... are
    all told apart, at and past the last row length the fp32 counts hold."""
    w = (m + 63) // 64
    words = np.full((5, w), np.uint64(0xFFFFFFFFFFFFFFFF), np.uint64)
    if m % 64:
        words[:, -1] = np.uint64((1 << (m % 64)) - 1)
    for r in range(5):
        words[r, :r] ^= np.uint64(1 << (7 * r))
    words[4, w // 3: w // 2] = np.uint64(0x5555555555555555)
    want, ws = ol.contig_matrix(words)
    c = sb.StormContig(m)
    c.set_schedule(sb.SCHED_TILES)
    c.add_bitmaps(words)
    got, s = c.matrix()
    np.testing.assert_array_equal(got, want)
    assert s == ws


@pytest.mark.parametrize("rows,universe", ((300, 65536 * 3 + 17), (513, 1 << 20), (200, (1 << 24) + 5)))
def test_gathered_rows(sb, rows, universe):
    """The row-mapped form: every row of a chunked container on the tensor
    cores, in one panel and in several, 4-bit and (past 2^24 values) 8-bit."""
    g = gen.rng(rows)
    sets = [np.unique(g.integers(0, universe, size=int(g.integers(1, 4000)))).astype(np.uint32) for _ in range(rows)]
    sets[rows // 2] = np.append(sets[rows // 2], np.uint32(universe - 1)) if universe - 1 not in sets[rows // 2] else \
        sets[rows // 2]
    vals, offs = gen.to_csr(sets)
    want, ws = ol.sets_matrix(vals, offs)
    for budget in (0, 512 * ((universe + 65535) // 65536) * 8256):
        s = sb.Storm()
        for v in sets:
            s.add(v)
        s.set_dense_block(1e-12, budget)
        got, total = s.matrix()
        np.testing.assert_array_equal(got, want)
        assert total == ws and s.last_dense()[0] == rows
        s.close()


@pytest.mark.parametrize("n,m", ((257, 513), (600, 65536), (300, 66049)))
def test_thresholded_form(sb, n, m):
    words = gen.bernoulli_rows(n, m, (0.2, 0.8), n + m)
    words[::5] = words[0]                                        # pairs of equal rows: Jaccard exactly 1
    tri, _ = ol.contig_matrix(words)
    c = sb.StormContig(m)
    c.add_bitmaps(words)
    for t in (0.0, 0.4, 1.0):
        wi, wj, wc = ol.threshold_pairs(tri, n, t)
        gi, gj, gc, found = c.threshold(t, cap=n * n)
        assert found == len(wi)
        np.testing.assert_array_equal(gi, wi)
        np.testing.assert_array_equal(gj, wj)
        np.testing.assert_array_equal(gc, wc)
