"""CPU test of the line bench.py prints: short enough for a reader that keeps the tail of the output, nothing that
describes the measured workload left out."""
import importlib.util
import json
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline", "parity")


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_line", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def full_line(bench):
    third = 1e6 / 3
    peaks = {"hbm_gbs": 6546.2, "fp8_tflops": 3330.6, "kind": "measured",
             "fp8_kind": "2 x measured bf16 burst (1665.3 TFLOP/s); no FP8 peak is measured on this pool"}
    name = "grouped_gemm_large_kernel<1>: GEMM1 + SwiGLU + plane split"
    roof = bench.roofline(name, 123456789012, 98765432109876, third, 864400000, peaks)
    parity = {"max_abs_over_rms": third, "cosine": 0.9999999674349365, "n": 29360128, "n_diff": 249018,
              "n_one_step": 223364, "n_multi_step": 25654, "match_ratio": 1.0, "max_abs_vs_f32_over_rms": third}
    stages = {k: third for k in ("route_permute", "gather", "gemm1", "swiglu_split", "gemm2", "combine")}

    def row(n, fast=False):
        return {"workload": n, "options": {"fast_combine": fast, "unfused": False}, "T": 4096, "n_sel": 5144,
                "active_experts": 26, "replicas": 6, "us_per_step": third, "tokens_per_s": third,
                "gpu_launches_per_step": 8, "split_k": [1, 1], "token_tile": [128, 128], "stage_us": stages,
                "roofline": roof, "whole_op": roof, "kernels": {"gemm1": roof, "gemm2": roof}, "parity": parity}
    head = row("decode_t1")
    return {"metric": bench.METRIC, "value": third, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": third, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "fp8_e4m3",
            "data": "synthetic", "config": bench.workload_config("decode_t1", 2, 2),
            "run_info": {"split_k": [0, 0], "token_tile": [16, 16], "replicas": 6},
            "e2e": {"value": third, "unit": bench.UNIT, "h2d_bytes_per_step": 8928, "d2h_bytes_per_step": 14336,
                    "ms_per_step": third, "note": "token tensors from pinned host memory, bf16 output read back; weights "
                    "stay resident"},
            "gpu_launches": 20, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [], "samples": 6},
            "roofline": roof, "whole_op": roof, "kernels": head["kernels"], "stage_us": stages,
            "cpu_baseline": {"kind": "port", "cores": 16, "value": third, "unit": bench.UNIT,
                             "sample": "50 calls of the oracle port on the same T=1 batch (3.8 s); only the experts the "
                             "batch uses are dequantised"},
            "parity": parity, "sweep": [row(n) for n in bench.WORKLOADS if n != "decode_t1"],
            "sweep_modes": [row("prefill_t4096", True), row("prefill_t4096")],
            "oracle_vs_oracle": dict(parity, what="oracle on GPU (fp32, TF32 off) vs oracle on CPU"),
            "scale_anchor": {"workload": "ep_layer_t16384", "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": third,
                             "tokens_per_s": third, "records": 64974, "parity": parity, "per_gpu": roof},
            "reference_cuda": {"unavailable": "oracle/_ref/libmoe_reference_cuda.so was not built (no reference checkout "
                               "at build time)"}}


def test_the_line_is_short_and_complete(bench, capsys, tmp_path):
    line = full_line(bench)
    bench.emit(line, str(tmp_path / "detail.json"))
    text = capsys.readouterr().out
    assert text.count("\n") == 1 and len(text) <= bench.LINE_LIMIT + 1
    out = json.loads(text)
    assert all(k in out for k in CONTRACT)
    for k in ("config", "clocks", "parity", "gpu_launches", "steps"):
        assert out[k] == bench._short(line[k])
    assert out["value"] == pytest.approx(line["value"], rel=1e-5)
    assert [r["workload"] for r in out["sweep"]] == [r["workload"] for r in line["sweep"]]
    assert all(r["us"] > 0 and r["match_ratio"] == 1.0 for r in out["sweep"])
    assert "scale_anchor" in out
    assert json.load(open(tmp_path / "detail.json")) == line
