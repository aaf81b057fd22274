"""The benchmark's JSON line stays short and complete, whatever its record holds."""
import json

import pytest

import bench

REQUIRED = ["metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "clocks", "gpu_launches"]


def _record(full):
    text = "words " * 100
    roof = {"kernel": text[:200], "bound": "int", "unit": "G Fp products/s", "ms": 38.23456789, "fp_products": 10 ** 12,
            "achieved": 21.23456789012345, "peak": 30.68921901788707, "frac": 0.7708650015274833, "traffic": None,
            "work_basis": text}
    section = {"value": 123456.789012345, "unit": "ciphertexts/s", "form": text, "ms_per_batch": 1.23456789012}
    sweep = {f"{k}_2^{lg}": dict(roof) for k in ("g1_msm", "g2_msm", "g1_ntt", "g2_ntt", "gt_ntt") for lg in range(8, 22, 2)}
    sweep["multi_pairing_k4096"] = dict(roof)
    return {
        "metric": bench.METRIC, "value": 213456.78901234567, "unit": "ciphertexts/s", "n_gpus": 8, "steps": 20,
        "warmup": 5, "ms_per_step": 923.4567890123456, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "u32 limbs (Fp/Fr Montgomery)", "data": "synthetic", "gpu_launches": 123456,
        "config": {"workload": "weighted_btx B=512 n=128 Zipf(1) W=4096 t=W/3", "batch_size": 512, "parties": 128,
                   "total_weight": 4096, "threshold": 1365, "committee": list(range(60)), "committee_weight": 1382,
                   "parallelism": "replicas x8", "form": text[:150], "l2": "flushed before every step (256 MB write)"},
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 3000},
        "roofline": roof, "rooflines": {f"kernel_{i}": roof for i in range(6)}, "roofline_plain": roof,
        "plain": section if full else {"value": None}, "plain_cached": section if full else {"value": None},
        "batched_graph": section, "cpu_baseline": {**section, "cores": 64, "kind": "port", "sample": text} if full else None,
        "e2e": {**section, "h2d_bytes_per_step": 314572800, "d2h_bytes_per_step": 113246208, "p50_ms": 41.0,
                "p99_ms": 112.25} if full else None,
        "wpfe_batched": {**section, "classes": {str(i): section for i in range(9)}} if full else None,
        "wpfe_served": section if full else None, "sweep": sweep if full else None, "setup_s": 33.0, "crs_load": {},
    }


@pytest.mark.parametrize("full", [True, False])
def test_the_line(full):
    record = _record(full)
    text = json.dumps(bench.headline(record))
    assert len(text) <= bench.HEADLINE_BYTES and "\n" not in text
    line = json.loads(text)
    assert [k for k in REQUIRED if k not in line] == []
    assert line["value"] == record["value"] and line["ms_per_step"] == record["ms_per_step"]
    if full:
        assert line["e2e"]["h2d_bytes_per_step"] == 314572800 and line["e2e"]["d2h_bytes_per_step"] == 113246208
        assert line["plain"] == 123456.8 and line["sweep_ms"]["g1_msm_2^16"] == 38.23457
