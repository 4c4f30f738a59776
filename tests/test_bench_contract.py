"""bench.py's reference arm (the CPU oracle port on the host cores) runs without a GPU and prints
the contract's JSON line: metric, unit, config and the cpu_baseline / e2e objects."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_prints_contract_line():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "1", "--cpu-tiles", "2"], capture_output=True, text=True, timeout=600,
                       cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e", "impl"):
        assert key in line, key
    assert line["impl"] == "reference" and line["value"] > 0 and line["higher_is_better"] is True
    assert line["unit"] == "tile-updates/s" and line["config"]["workload"] == "tlr_gemm_n16384_nb512"
    cb = line["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["value"] == line["value"]
    assert line["e2e"]["value"] == line["value"]
    assert line["e2e"]["h2d_bytes_per_step"] == 0 and line["e2e"]["d2h_bytes_per_step"] == 0


def _full_block(n_forms, note):
    clocks = {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 62}
    forms = {f"form_{i}_ff48": {"value": 12345.678901234567 + i, "unit": "tile-updates/s", "note": note, "clocks": clocks,
                                "e2e": {"value": 11345.678901234567, "unit": "tile-updates/s"}} for i in range(n_forms)}
    return {"metric": "TLR-GEMM tile-updates/s at 1e-8 rel err: plain FP64 vs batched mixed+learned",
            "value": 53467.12033798017, "unit": "tile-updates/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 612.8626302083334, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic (Morton-sorted exponential kernel, seeded)",
            "config": {"workload": "tlr_gemm_n16384_nb512", "n": 16384, "nb": 512, "tiles": "32x32",
                       "updates_per_step": 32768, "accuracy": 1e-8, "threshold": "relative", "form": "plain_fp64",
                       "parallelism": "single_gpu", "l2": "inputs larger than L2, no flush", "launch_shapes": {"note": note}},
            "e2e": {"value": 52599.3162992059, "unit": "tile-updates/s", "h2d_bytes_per_step": 541761536,
                    "d2h_bytes_per_step": 309891080, "transfer": note},
            "roofline": {"bound": "fp64", "kernel": "qr", "achieved": 0.6, "peak": 1.06, "unit": "TFLOP/s",
                         "frac": 0.57, "note": note},
            "gpu_launches": 133140, "check": {"rel_fro_err_vs_fp64_dense_product": 2.4381832571859275e-08},
            "parity": {"rank_violations": 0, "bar": note}, "forms": forms,
            "cpu_baseline": {"value": 6434.168814342794, "cores": 16, "kind": "port", "sample": note}, "clocks": clocks}


def test_own_arm_prints_a_short_line(capsys, tmp_path):
    """Whatever the blocks hold, the printed line is short and has the contract's keys; the file has everything."""
    sys.path.insert(0, ROOT)
    import bench
    for n_forms, note in ((4, "x" * 2000), (60, "y" * 9000)):
        full = _full_block(n_forms, note)
        path = tmp_path / "details.json"
        bench.emit(full, str(path))
        out = capsys.readouterr().out
        assert out.count("\n") == 1 and len(out) <= 1401
        line = json.loads(out)
        for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                    "scaling", "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
            assert key in line, key
            if key not in ("config", "e2e", "clocks"):
                assert line[key] == full[key], key
        for key, sub in (("config", "workload"), ("config", "l2"), ("e2e", "value"), ("e2e", "unit"),
                         ("e2e", "h2d_bytes_per_step"), ("e2e", "d2h_bytes_per_step"), ("clocks", "sm_mhz"),
                         ("clocks", "sm_max_mhz"), ("clocks", "reasons")):
            assert line[key][sub] == full[key][sub], (key, sub)
        assert json.loads(path.read_text()) == full
