"""What the benchmark prints about itself, without a GPU."""
import importlib

import pytest


@pytest.fixture(scope="module")
def bench():
    return importlib.import_module("bench")


def test_tensor_peak_is_the_pipe_at_the_sampled_clock(bench, monkeypatch):
    import torch

    class Props:
        multi_processor_count = 148

    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: Props)
    at = {mhz: bench.tensor_peak_tops(0, True, mhz)[0] for mhz in (1000.0, 1790.0)}
    # 65536 operations a clock and CTA pair, 74 pairs
    assert at[1000.0] == pytest.approx(65536 * 74 * 1000e6 / 1e12)
    assert at[1790.0] == pytest.approx(1.79 * at[1000.0])
    # the kernel's profile: 8050 TOPS at 92.8 % pipe activity, which no bound may be under
    assert at[1790.0] > 8050
    assert bench.tensor_peak_tops(0)[0] >= at[1790.0]
