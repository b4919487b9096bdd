"""How the postings' passes deal rows to warps, checked without a GPU
(tests/walk_check.cu): every chunk once, and few items that find none."""
from harness import run_host_check


def test_walk_items(sb):
    assert run_host_check("walk_check").strip().endswith("ok")
