"""bench.py's reference arm on the host cores: one JSON line with the keys
of the benchmark contract (run on the small 32^3 workload so that it ends
in seconds)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


def test_reference_arm_prints_the_contract_line():
    from oracle import build
    if not os.path.exists(build.ref_lib_path(32)) and not build.reference_available():
        pytest.skip("reference build unavailable")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--config", "tiny", "--steps", "2",
                        "--warmup", "1"], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [ln for ln in r.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
              "scaling", "vs_baseline", "dtype", "data", "config", "impl", "cpu_baseline", "e2e"):
        assert k in d, k
    assert d["impl"] == "reference" and d["steps"] == 2 and d["warmup"] == 1
    assert d["value"] > 0 and d["ms_per_step"] > 0 and d["higher_is_better"] is True
    assert d["config"]["workload"].startswith("tiny32")
    cb = d["cpu_baseline"]
    assert cb["kind"] == "reference" and cb["cores"] >= 1 and cb["value"] == d["value"] and cb["sample"]
    assert d["e2e"] == {"value": d["value"], "unit": d["unit"], "h2d_bytes_per_step": 0,
                        "d2h_bytes_per_step": 0}


def test_reference_arm_without_the_reference():
    """Without ARGOT's sources or a library built from them the arm says so
    in its one line and ends well."""
    from oracle import build
    if os.path.exists(build.ref_lib_path(32)) or build.reference_available():
        pytest.skip("the reference is at hand")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--config", "tiny"], cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(ln) for ln in r.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and lines[0]["unavailable"]


@pytest.mark.gpu
def test_our_arm_without_the_reference(cuda_ok):
    """Our arm prints its line whether or not the reference is at hand; the
    parity block names what it compared with."""
    r = subprocess.run([sys.executable, "bench.py", "--config", "tiny", "--steps", "2", "--warmup", "3"], cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(ln) for ln in r.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    d = lines[0]
    assert d["value"] > 0 and d["e2e"]["value"] > 0 and d["gpu_launches"] > 0
    p = d["parity"]
    assert "O1" in p["oracle"]
    assert p["reference_order"]["ray_lists_equal_O1"] and p["reference_order"]["columns_bitwise_O1"]
    assert max(p["exact_f32_vs_fp64"].values()) < 1e-4
