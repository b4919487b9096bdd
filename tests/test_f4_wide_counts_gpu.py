"""The 4-bit tensor-core kernel's drain of blocks that hold a count past 65535:
the 16-bit counts a warp has packed are dropped and the block is stored from
tensor memory through the same shared-memory words, 32 bits each. Tiles with
such blocks beside blocks that stay packed, every count different from its
neighbours'. Whole numbers, equal to the oracle's."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu

M = 140032     # bits: pairs of rows of density 0.9 share about 113000, of 0.3 and 0.9 about 38000


def _rows(n):
    """Dense and sparse rows by turns of 40, so that 32-row blocks hold both, some one kind only."""
    words = gen.bernoulli_rows(n, M, (0.1, 0.4), n)
    dense = gen.bernoulli_rows(n, M, (0.8, 1.0), n + 1)
    pick = (np.arange(n) // 40) % 3 == 1
    words[pick] = dense[pick]
    return words


@pytest.mark.parametrize("n", (31, 130, 300))
def test_blocks_past_16_bits(sb, n):
    words = _rows(n)
    words[n // 2] = gen.bernoulli_rows(1, M, 1.1, 1)[0]
    want, ws = ol.contig_matrix(words)
    assert (want > 65535).any() and (want < 65536).any()
    for sched in (sb.SCHED_TILES, sb.SCHED_STREAM_K):
        c = sb.StormContig(M)
        c.set_schedule(sched)
        c.add_bitmaps(words)
        got, s = c.matrix()
        np.testing.assert_array_equal(got, want, err_msg=str(sched))
        assert s == ws
        c.close()


def test_gathered_blocks_past_16_bits(sb):
    """The same through a row map, by the chunked container's tensor rows."""
    n = 300
    words = _rows(n)
    bits = np.unpackbits(words.view(np.uint8), axis=1, bitorder="little")
    sets = [np.flatnonzero(b).astype(np.uint32) for b in bits]
    want, ws = ol.contig_matrix(words)
    s = sb.Storm()
    for v in sets:
        s.add(v)
    s.set_dense_block(1e-12)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws and s.last_dense()[0] == n
    s.close()


@pytest.mark.parametrize("m", (1 << 24, (1 << 24) - 4097))
def test_large_counts_of_random_rows(sb, m):
    """Counts near 2^24 that grow by irregular steps all the way (dense random
    rows), whole tiles and K segments added up: every step of the fp32 counts is
    a whole number below 2^24, exact."""
    w = (m + 63) // 64
    g = gen.rng(m)
    words = ~(g.integers(0, 1 << 64, size=(9, w), dtype=np.uint64) & g.integers(0, 1 << 64, size=(9, w), dtype=np.uint64)
              & g.integers(0, 1 << 64, size=(9, w), dtype=np.uint64) & g.integers(0, 1 << 64, size=(9, w), dtype=np.uint64))
    words[3] |= ~np.uint64(0)                                    # a full row: counts equal the others' sizes
    if m % 64:
        words[:, -1] &= np.uint64((1 << (m % 64)) - 1)
    want, ws = ol.contig_matrix(words)
    for sched in (sb.SCHED_TILES, sb.SCHED_STREAM_K):
        c = sb.StormContig(m)
        c.set_schedule(sched)
        c.add_bitmaps(words)
        got, s = c.matrix()
        np.testing.assert_array_equal(got, want, err_msg=str(sched))
        assert s == ws
        c.close()
