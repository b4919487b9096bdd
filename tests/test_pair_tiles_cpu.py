"""Tiles and host-call plans of the CTA-pair kernels, checked without a GPU
(tests/pair_tiles_check.cu)."""
import pytest

from harness import run_host_check


@pytest.mark.timeout(600)
def test_pair_tiles_and_host_plan(sb):
    assert run_host_check("pair_tiles_check").strip().endswith("ok")
