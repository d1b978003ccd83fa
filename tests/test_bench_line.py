"""bench.py's printed line stays short (a reader may keep only the end of the
output) whatever its sections hold, and keeps the numbers that are compared."""
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))


def _stats(x):
    return {"qps": 34567.123456789 * x, "p50_ms": 0.123456789012, "p99_ms": 1.23456789012, "light_p50_ms": 0.123456789012,
            "light_p99_ms": 1.23456789012, "heavy_p50_ms": 0.123456789012, "heavy_p99_ms": 1.23456789012,
            "mean_batch": 4.895061728395062, "failed": 0}


def test_line_is_short():
    import bench
    cdf = [0.123456789012345] * 25
    types = {f"light_q{i}": {"weight": 2800, "heavy": False, "completed": 5483, "failed": 0, "qps": 1.0 / 3, "p50_ms": 1.0 / 3,
                             "p99_ms": 2.0 / 3, "cdf_ms": cdf} for i in range(10)}
    line = {"metric": "m", "value": 1803.123456789, "e2e": {"value": 97.123456789}, "roofline": {"frac": 1.0 / 3},
            "per_op": [{"op": i, "ms_mean": 1.0 / 3, "achieved": 2.0e3 / 3, "kind": "k2u"} for i in range(12)],
            "paged": {"configs": [{"budget": 1.0 / 3, "qps": 2.0e3 / 3}] * 8},
            "serving": {"config": "c" * 230, "baseline_capacity_qps": 2.0e4 / 3,
                        "sweep": [{"rate_qps": 2.0e4 / 3 * f, "query_at_a_time_stats": _stats(f) if f < 2 else None,
                                   "batched_learned": _stats(f)} for f in range(1, 14)],
                        "headline": {"baseline_qps": 2.0e4 / 3, "ratio": 23.0 / 3, "cdf_rates": cdf,
                                     "baseline_cdf_ms": {"light": cdf, "heavy": cdf},
                                     "batched_cdf_ms": {"light": cdf, "heavy": cdf},
                                     "baseline_per_type": types, "batched_per_type": types}}}
    full = json.dumps(line)
    out = json.loads(json.dumps(bench.brief(line)))
    assert json.loads(full) == line                       # the line itself is left as it was
    assert len(json.dumps(out)) < 6000 < len(full)
    assert out["value"] == line["value"] and out["e2e"] == line["e2e"] and out["roofline"] == line["roofline"]
    s = out["serving"]
    assert abs(s["headline"]["ratio"] - 23.0 / 3) < 1e-4
    assert len(s["sweep"]) == 13 and s["sweep"][4][1] is None
    assert len(s["sweep"][4][2]) == len(s["sweep_columns"])
    assert "cdf" not in json.dumps(out)
