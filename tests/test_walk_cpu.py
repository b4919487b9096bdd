"""How the postings' passes deal rows to warps, checked without a GPU
(tests/walk_check.cu): every chunk once, and few items that find none."""
from harness import run_host_check


def test_walk_items(sb):
    assert run_host_check("walk_check").strip().endswith("ok")


def test_rows_by_value_count(sb):
    """The planner's order of the rows (tests/row_order_check.cu): made when it
    is first asked for after an upload, not for the calls that do without it; and
    the memory that a wider panel needs."""
    assert run_host_check("row_order_check").strip().endswith("ok")
