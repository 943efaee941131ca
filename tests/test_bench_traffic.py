"""bench.py pairs a query's time only with DRAM bytes captured from a form of as many kernels."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_traffic_of_another_form_is_left_out(tmp_path, monkeypatch):
    import bench
    (tmp_path / "profiles").mkdir()
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench._profiled_traffic("q.json", 17) is None
    for kernels, want in ((17, 123), (16, None), (None, None)):
        d = {"dram_bytes_per_launch": 123}
        if kernels:
            d["kernels"] = kernels
        (tmp_path / "profiles" / "q.json").write_text(json.dumps(d))
        assert bench._profiled_traffic("q.json", 17) == want


def test_committed_profiles_are_of_the_present_form():
    import bench
    assert bench._profiled_traffic("cc_query_ba1m.json", bench.KERNELS_PER_QUERY)
    assert bench._profiled_traffic("cc_filter_ba1m.json", 1)
