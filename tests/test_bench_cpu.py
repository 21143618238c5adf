"""The benchmark's contract on a machine without a GPU: the reference arm falls back to the CPU oracle and still
prints one JSON line with the agreed keys; the native arm refuses to run (no CPU fallback in the product)."""
import importlib.util
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _no_gpu():
    try:
        import torch
        return not torch.cuda.is_available()
    except Exception:
        return True


@pytest.mark.skipif(not _no_gpu(), reason="checks the behaviour without a GPU")
def test_reference_arm_falls_back_to_the_cpu_oracle():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "3", "--warmup", "3",
                        "--seq", "64"], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    line = [l for l in r.stdout.splitlines() if l.startswith("{")][-1]
    d = json.loads(line)
    assert d["impl"] == "reference" and d["unit"] == "sequences/s" and d["higher_is_better"] is True
    assert d["value"] > 0 and d["cpu_baseline"]["kind"] == "port" and d["cpu_baseline"]["cores"] >= 1
    assert d["e2e"]["h2d_bytes_per_step"] == 0 and d["e2e"]["d2h_bytes_per_step"] == 0
    assert "workload" in d["config"]


@pytest.mark.skipif(not _no_gpu(), reason="checks the behaviour without a GPU")
def test_native_arm_has_no_cpu_fallback():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--steps", "3", "--warmup", "3"],
                       capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode != 0
    assert "no CPU fallback" in (r.stderr + r.stdout)


@pytest.mark.parametrize("stages,stage_bytes,kernel", [(3, 26624, "tile_gemm_kernel"), (0, 0, "resident_kernel"), (1, 0, "dense_kernel"), (4, 0, "dense_split_kernel")])
def test_roofline_names_the_kernel_that_a_weight_runs_in(stages, stage_bytes, kernel):
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    assert bench.linear_kernel({"stages": stages, "stage_bytes": stage_bytes}) == kernel
