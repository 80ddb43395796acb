"""The bench's roofline entry of the finest sweep: the FP32 sweep, whose u stays in
L2, is compared with the HBM peak by its DRAM traffic and not by the bytes that
it moves through L2; a size without a traffic record has no HBM fraction."""
import importlib
import json
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def bench(monkeypatch):
    monkeypatch.syspath_prepend(ROOT)
    m = importlib.import_module("bench")
    monkeypatch.setattr(m, "measured_peaks", lambda: (6800.0, "measured"))
    return m


def _profile(n, words, size, ms):
    return {"relax_calls": 10, "relax_ms": 10 * ms, "relax_bytes": 10.0 * words * size * (n + 2) ** 3,
            "relax_bits": 8 * size}


def test_fp32_sweep(bench):
    with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
        dram = json.load(f)["k_relax32_split@256"]["dram_bytes_per_launch"]
    r = bench.relax_roofline(_profile(256, 4, 4, 0.044), 9.5, 256)
    assert r["bound"] == "l2" and r["traffic"] == dram
    assert r["achieved"] == pytest.approx(dram / 44e-6 / 1e9)
    assert r["frac"] == pytest.approx(r["achieved"] / 6800.0) and r["frac"] < 0.5
    assert r["l2_gbs"] == pytest.approx(16 * 258 ** 3 / 44e-6 / 1e9) and "16 B/cell" in r["kernel"]
    r = bench.relax_roofline(_profile(48, 6, 4, 0.006), 1.0, 48)
    assert r["achieved"] is None and r["frac"] is None and r["l2_gbs"] > 0 and "24 B/cell" in r["kernel"]


def test_fp64_sweep(bench):
    r = bench.relax_roofline(_profile(256, 6, 8, 0.26), 40.0, 256)
    assert r["bound"] == "fp64" and r["l2_gbs"] is None and "at most 48 B/cell" in r["kernel"]
    assert r["achieved"] == pytest.approx(48 * 258 ** 3 / 0.26e-3 / 1e9)
    r = bench.relax_roofline({"relax_calls": 0, "relax_ms": 0.0, "relax_bytes": 0.0, "relax_bits": 64}, 0.0, 64)
    assert r["achieved"] is None and r["frac"] is None and r["share_of_step"] is None
