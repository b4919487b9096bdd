"""The row walks of the chunked engine -- postings, run postings, expansion to
bitmaps, transposed panel -- on rows at the edges of their groups: chunks of no
more than a few values (walked 32 at a time) in rows of more and fewer than 32
chunks, missing chunk ids, lists around multiples of 8 and 256 entries, runs
across those steps and across bins. Whole numbers, equal to the oracle's."""
import numpy as np
import pytest

import gen
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _short(g):
    """1 to 5 values in some of 70 chunks: groups of 32 chunks, the last one partial."""
    sets = []
    for r in range(150):
        ids = np.flatnonzero(g.random(70) < (0.2, 0.9, 1.0)[r % 3])
        v = [int(c) << 16 | int(x) for c in ids for x in g.integers(0, 40, size=int(g.integers(1, 6)))]
        sets.append(np.unique(np.array(v, dtype=np.uint32)))
    return sets


def _lists(g):
    """One to three chunks of 1 .. 4095 values, lengths around 8, 256 and 2048."""
    sizes = (1, 7, 8, 9, 255, 256, 257, 263, 511, 513, 2047, 2048, 2049, 4095)
    sets = []
    for r in range(84):
        v = [np.sort(g.choice(65536, size=sizes[(r + k) % len(sizes)], replace=False)) + (int(c) << 16)
             for k, c in enumerate(np.sort(g.choice(9, size=1 + r % 3, replace=False)))]
        sets.append(np.concatenate(v).astype(np.uint32))
    return sets


def _runs(g):
    """Runs of 1 .. 700 values, adjacent ones and ones that end at a chunk's last value included."""
    sets = []
    for r in range(90):
        v = [np.arange(s, s + int(g.integers(1, 700))) for s in g.integers(0, 5 * 65536 - 700, size=int(g.integers(1, 14)))]
        v.append(np.arange(65536 - int(g.integers(1, 300)), 65536))
        v.append(np.arange(65536, 65536 + int(g.integers(1, 300))))
        sets.append(np.unique(np.concatenate(v)).astype(np.uint32))
    return sets


def _mixed(g):
    """Bitmap chunks, long and short lists in the same rows, chunks missing."""
    sets = []
    for r in range(60):
        v = []
        for c in np.flatnonzero(g.random(40) < 0.5):
            n = int((3, 300, 4095, 9000)[int(g.integers(0, 4))])
            v.append(np.sort(g.choice(65536, size=n, replace=False)) + (int(c) << 16))
        sets.append(np.concatenate(v).astype(np.uint32) if v else np.array([5], np.uint32))
    return sets


CORPORA = {"short": _short, "lists": _lists, "runs": _runs, "mixed": _mixed}
# forced engines: postings list by list / row sweep / run sweep, transposed panel, tensor rows, the planner's choice
MODES = ("lists", "rows", "runs", "panel", "tensor", "auto")


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("corpus", sorted(CORPORA))
def test_walks_match_oracle(sb, corpus, mode):
    sets = CORPORA[corpus](gen.rng(len(corpus) * 7 + 1))
    vals, offs = gen.to_csr(sets)
    want, ws = ol.sets_matrix(vals, offs)
    s = sb.Storm()
    s.add_rows(vals, offs)
    if mode in ("lists", "rows", "runs"):
        s.set_panel(0)
        s.set_sparse_postings({"lists": 2, "rows": 3, "runs": 4}[mode])
    elif mode == "panel":
        s.set_panel(2)
    elif mode == "tensor":
        s.set_dense_block(1e-12)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws
    assert s.pairw_intersect_cardinality() == ws
    other = sb.Storm()
    other.add_rows(vals, offs)
    assert s.square(other) == 2 * ws + int(sum(len(v) for v in sets))
    s.close()
    other.close()


@pytest.mark.parametrize("universe", (1 << 20, (1 << 27) + 12345, 1 << 30))
def test_zone_maps_of_row_blocks(sb, universe):
    """Kernel-layer blocks whose rows' occupancy is folded in shared memory and
    (past 2^27 values) converted row by row: clustered rows, most tiles rejected."""
    g = gen.rng(11)
    sets = [np.unique((int(g.integers(0, 8)) * (universe // 8) + g.integers(0, 3000, size=600)).clip(max=universe - 1))
            .astype(np.uint32) for _ in range(200)]
    vals, offs = gen.to_csr(sets)
    _, ws = ol.sets_matrix(vals, offs)
    r = sb.StormRows(universe)
    r.set_bitmap_budget(0)
    for v in sets:
        r.add(v)
    assert r.allpairs_sum(sb.POLICY_PERTILE, 32)[0] == ws
    assert r.allpairs_sum(sb.POLICY_PERTILE, 64)[0] == ws
    r.close()


@pytest.mark.parametrize("n", (2, 511, 513, 3001))
def test_row_sweep_in_16_bits(sb, n):
    """The row sweep over 16-bit lists: values of one row and of all rows (the
    longest list), empty rows, an odd number of counters, beside chunk-kernel
    rows that leave gaps in the rows' order."""
    g = gen.rng(n)
    sets = [np.unique(np.concatenate([g.integers(0, 3 << 16, size=int(g.integers(0, 60))), [7, 70000]])).astype(np.uint32)
            for _ in range(n)]
    sets[0] = np.array([7, 70000, 123456], np.uint32)
    if n > 2:
        sets[n // 2] = np.zeros(0, np.uint32)
    for dup in (False, True):
        rows = list(sets)
        if dup:
            rows[n - 1] = np.sort(np.concatenate([rows[n - 1], rows[n - 1][:1]]))
        vals, offs = gen.to_csr(rows)
        want, ws = (ol.storm_matrix if dup else ol.sets_matrix)(vals, offs)
        s = sb.Storm()
        for v in rows:
            s.add(v)
        s.set_dense_block(0.0)
        s.set_panel(0)
        s.set_sparse_postings(3)
        got, total = s.matrix()
        strict = np.not_equal(*np.triu_indices(n))
        np.testing.assert_array_equal(got[strict], want[strict])
        assert total == ws
        s.close()


@pytest.mark.parametrize("n", (2, 300, 52000))
def test_outputs_that_held_other_values(sb, n):
    """Every entry of the triangle is written, whatever the buffer held: row
    sweeps over all rows (no clear before them; past 65535 x 16 bits and one
    block of counters too), the list form, and empty rows."""
    import torch

    g = gen.rng(n)
    card = g.integers(0, 12, size=n) if n < 1000 else (np.arange(n) % 1000 == 0) * 9
    base = g.integers(0, 1 << 18, size=n)
    sets = [np.unique(base[r] % 3 * 70000 + g.integers(0, 50, size=int(card[r]))).astype(np.uint32) for r in range(n)]
    if n > 1000:                                # one row past 16 bits, in list chunks: counters of 32 bits
        sets[n - 1] = (np.arange(0, 65536, 17)[None, :] + (np.arange(20) << 16)[:, None]).ravel().astype(np.uint32)
    vals, offs = gen.to_csr(sets)
    out = torch.empty(n * (n + 1) // 2, dtype=torch.int32, device="cuda")
    s = sb.Storm()
    s.add_rows(vals, offs)
    s.set_dense_block(0.0)
    s.set_panel(0)
    got = []
    for mode in (2, 3, 4):
        s.set_sparse_postings(mode)
        out.fill_(-7)
        s.matrix_device(out.data_ptr(), out.numel())
        torch.cuda.synchronize()
        got.append(out.clone())
    s.close()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    if n < 1000:
        want, _ = ol.sets_matrix(vals, offs)
        np.testing.assert_array_equal(got[0].cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("n", (1, 512, 513, 1024, 1025, 2049))
def test_panel_widths_and_counter_flushes(sb, n):
    """Transposed blocks of 512, 1024 and 2048 rows (and one row in a second
    block), queried by rows of fewer values than a batch, of more than the
    counters hold between two flushes (2016 words), in one work item and in
    several, lists and bitmap chunks in one row, chunks missing, empty rows."""
    g = gen.rng(n)
    sets = []
    for r in range(n):
        v = [g.integers(0, 1 << 22, size=int(g.integers(0, 40))), np.arange(r % 7, 50)]
        if r % 64 == 1:
            v.append(g.integers(0, 40 << 16, size=30000))          # list chunks, split into items
        if r % 100 == 3:
            v.append((5 << 16) + g.choice(65536, size=9000, replace=False))   # a bitmap chunk
        sets.append(np.unique(np.concatenate(v)).astype(np.uint32))
    sets[n // 2] = np.zeros(0, np.uint32)
    vals, offs = gen.to_csr(sets)
    want, ws = ol.sets_matrix(vals, offs)
    s = sb.Storm()
    s.add_rows(vals, offs)
    s.set_panel(2)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws and s.last_panel_rows() in (0, n)
    s.close()
