"""Which engine and which form of the postings a forced call takes, and the
limits at which the row sweep changes its kernel: 65535 rows and 65535 values
(members, lengths and counts of 16 bits), and partners in two blocks past that.
Whole numbers, equal to the oracle's or to counts known from how the rows are
made."""
import numpy as np
import pytest

import gen
import oracle_lib as ol
from test_storm_t_walks_gpu import _lists, _runs, _short

pytestmark = pytest.mark.gpu

FORMS = {2: 0, 3: 1, 4: 2}     # set_sparse_postings mode -> last_postings_form


def _storm(sb, sets, mode):
    vals, offs = gen.to_csr(sets)
    s = sb.Storm()
    s.add_rows(vals, offs)
    s.set_dense_block(0.0)
    s.set_panel(0)
    s.set_sparse_postings(mode)
    return s


@pytest.mark.parametrize("corpus", (_short, _lists, _runs))
def test_forced_forms_run(sb, corpus):
    sets = corpus(gen.rng(17))
    want, ws = ol.sets_matrix(*gen.to_csr(sets))
    for mode, form in FORMS.items():
        s = _storm(sb, sets, mode)
        got, total = s.matrix()
        np.testing.assert_array_equal(got, want, err_msg=str(mode))
        assert total == ws
        assert s.last_postings_form() == form and s.last_postings_rows() == len(sets)
        s.close()


@pytest.mark.parametrize("n", (2, 512, 513, 1025, 2049))
def test_forced_panel_holds_every_row(sb, n):
    g = gen.rng(n)
    sets = [np.unique(g.integers(0, 1 << 20, size=int(g.integers(0, 50)))).astype(np.uint32) for _ in range(n)]
    want, ws = ol.sets_matrix(*gen.to_csr(sets))
    s = sb.Storm()
    s.add_rows(*gen.to_csr(sets))
    s.set_panel(2)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws and s.last_panel_rows() == n and s.last_postings_form() == -1
    s.close()


@pytest.mark.parametrize("n", (2, 511, 3001))
def test_row_sweep_writes_the_diagonal(sb, n):
    g = gen.rng(n)
    sets = [np.unique(np.concatenate([g.integers(0, 3 << 16, size=int(g.integers(0, 60))), [7, 70000]])).astype(np.uint32)
            for _ in range(n)]
    want, ws = ol.sets_matrix(*gen.to_csr(sets))
    s = _storm(sb, sets, 3)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws and s.last_postings_form() == 1
    s.close()


@pytest.mark.parametrize("values", (65535, 65536))
def test_row_sweep_of_long_equal_rows(sb, values):
    """Counts at and past 16 bits, in list chunks."""
    x = ((np.arange(17, dtype=np.uint32)[:, None] << 16) + np.arange(0, 65536, 17, dtype=np.uint32)[None, :]).ravel()[:values]
    assert len(x) == values
    sets = [x, x[::2].copy(), x, np.zeros(0, np.uint32), x[:1].copy()]
    want, ws = ol.sets_matrix(*gen.to_csr(sets))
    s = _storm(sb, sets, 3)
    got, total = s.matrix()
    np.testing.assert_array_equal(got, want)
    assert total == ws and s.last_postings_form() == 1
    s.close()


@pytest.mark.parametrize("n", (65535, 65536))
def test_row_sweep_at_the_limit_of_its_rows(sb, n):
    """Row r holds 5, 100 + r % 50 and 70000 + r % 33: the counts are known. Value
    5 has a list of every row."""
    import torch

    r = np.arange(n, dtype=np.uint32)
    vals = np.stack([np.full(n, 5, np.uint32), 100 + r % 50, 70000 + r % 33], axis=1).ravel().astype(np.uint32)
    s = sb.Storm()
    s.add_rows(vals, np.arange(0, 3 * n + 1, 3, dtype=np.uint64))
    s.set_dense_block(0.0)
    s.set_panel(0)
    s.set_sparse_postings(3)
    out = torch.full((n * (n + 1) // 2,), -7, dtype=torch.int32, device="cuda")
    total = s.matrix_device(out.data_ptr(), out.numel())
    torch.cuda.synchronize()
    assert s.last_postings_form() == 1 and s.last_postings_rows() == n
    s.close()
    a = torch.arange(n, device="cuda") % 50
    b = torch.arange(n, device="cuda") % 33
    at, bad, ws = 0, 0, 0
    for i in range(n):
        want = 1 + (a[i:] == a[i]).int() + (b[i:] == b[i]).int()
        bad += (out[at:at + n - i] != want).sum()
        ws += want[1:].sum()
        at += n - i
    assert int(bad) == 0 and total == int(ws)
