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


def test_line_is_short_whatever_the_forms(bench, tmp_path):
    import json

    line = {"metric": bench.METRIC, "value": 1.0, "roofline": {"frac": 0.93, "peak": 8700.0}, "e2e": {"value": 2.0}}
    forms = {"storm_t_full": {f"c{k}": {"device": {"pairs_per_s": 1e9 + k, "ms": 3.0}, "checked": {"identities_hold": True},
                                        "notes": "x" * 2000} for k in range(6)},
             "config5a_full": {"pairs_per_s": 2e11, "roofline": {"frac": 0.9}}, "form_seconds": {}}
    path = tmp_path / "out" / "forms.json"
    text = bench.report(line, forms, str(path))
    assert len(text) < 8000 and "\n" not in text
    got = json.loads(text)
    assert {k: got[k] for k in line} == line
    assert got["summary"]["c3"]["ms"] == 3.0 and got["summary"]["headline_frac"] == 0.93
    assert json.loads(path.read_text()) == forms
    assert "forms_file" not in json.loads(bench.report(line, {}, str(tmp_path / "none.json")))
