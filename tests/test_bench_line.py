"""The bench's result line: its figures whole, its details left out, short
enough for the end of a log that keeps a few thousand characters."""

from __future__ import annotations

import json

import bench


def test_short_line_keeps_the_figures():
    text = "x" * 100
    latency = {f"{p}%": {"p99_ms": 1.23456789, "requests": 9672, "by": {c: 0.123456789 for c in "ABCDEFGH"}}
               for p in (10, 30, 50, 70, 90, 100)}  # fmt: skip
    demapper = {"results": {f"qam{o}_{m}": {"us": 22.8159993, "gbs": 4412.1, "err": {"max_abs": 1e-5}, "text": text}
                            for o in (16, 64, 128) for m in ("maxlog", "exact")}}  # fmt: skip
    single = {"value": 1.8596813723, "e2e": {"value": 1.57143, "form": text}, "roofline": {"text": text * 5}}
    line = {
        "metric": bench.METRIC, "value": 4.1403401131948385, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 3.4659413496653237, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic (seeded)", "config": {"workload": text * 2, "l2": text, "form": text},
        "e2e": {"value": 3.8362233622958524, "unit": bench.UNIT, "h2d_bytes_per_step": 79577856,
                "d2h_bytes_per_step": 148062304, "form": text * 3, "with_copies": {"form": text}},
        "gpu_launches": 20, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "window": text},
        "plain": {"value": 3.4, "ms_per_step": 4.2, "bit_identical_to_batched": True, "form": text},
        "parity": {"frames_checked": 48, "bit_exact": True, "decoder_vs_fp64": {"text": text * 6}},
        "roofline": {"kernel": text, "bound": "smem", "achieved": 9866.56, "peak": 40273.92, "unit": "GB/s",
                     "frac": 0.245, "hbm": {"text": text * 4}},
        "configs": {"3": single, "1": single, "2": demapper, "2_mpoint": demapper,
                    "5": {"saturation": {"gbps": 3.24}, "latency_vs_load": latency,
                          "feed": {"oldest": {"p99_ms_at_70pct": 3.8, "latency_vs_load": latency}}},
                    "f1_montecarlo": {"error": "RuntimeError: " + text * 3}},
    }  # fmt: skip
    out = bench.short_line(line)
    assert len(json.dumps(out)) < 3000 < len(json.dumps(line))
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks"):  # fmt: skip
        assert out[key] == line[key]
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert out["e2e"][key] == line["e2e"][key]
    assert out["parity"] == {"frames_checked": 48, "bit_exact": True}
    assert out["configs"]["3"] == {"gbps": 1.8597, "e2e_gbps": 1.5714}
    assert out["configs"]["2"]["qam16_maxlog_us"] == 22.816
    assert out["configs"]["5"]["p99_ms"]["70%"] == 1.2346
    assert out["configs"]["f1_montecarlo"]["error"].startswith("RuntimeError")
