"""The benchmark's JSON contract, checked on the CPU through the reference arm (no GPU needed)."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm_prints_one_contract_line():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                          "--warmup", "0"], capture_output=True, text=True, timeout=600, check=True).stdout
    lines = [ln for ln in out.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    for k in ("impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
              "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert k in d, k
    assert d["impl"] == "reference" and d["unit"] == "tokens/s" and d["higher_is_better"] is True
    assert "workload" in d["config"] and d["vs_baseline"] is None
    assert d["cpu_baseline"]["kind"] in ("port", "reference") and d["cpu_baseline"]["cores"] >= 1
    assert d["e2e"]["h2d_bytes_per_step"] == 0 and d["e2e"]["d2h_bytes_per_step"] == 0
    assert d["value"] > 0 and abs(d["e2e"]["value"] - d["value"]) < 1e-9 * d["value"] + 1e-9


def test_reference_arm_is_silent_on_other_ranks():
    env = dict(os.environ, RANK="1", WORLD_SIZE="2", LOCAL_RANK="1")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2",
                        "--steps", "1", "--warmup", "0"], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0
    assert not [ln for ln in r.stdout.splitlines() if ln.startswith("{")]


def test_kernel_names_follow_the_library_s_choice():
    """At head size 64 unpacked rows and packed bf16 ones run in chunks at every size; packed fp32 ones, and fp32 ones at 32, while all
    sequences are resident."""
    import bench
    name = lambda sequences, **wl: bench.backward_kernel(dict(dict(E=64, dtype="bf16"), **wl), sequences)
    assert name(16384, op="srwm") == ("srwm_bwd2_kernel", False)
    assert name(256, op="srwm", E=32, dtype="f32") == ("srwm_bwd_kernel", False)
    assert name(8192, op="delta") == ("delta_bwd_chunk_kernel", True)
    assert name(256, op="delta", dtype="f32") == ("delta_bwd_chunk_kernel", True)
    assert name(512, op="delta", dtype="f32", E=32) == ("delta_bwd_kernel", False)
    assert name(148, op="delta", dtype="f32") == ("delta_bwd_chunk_kernel", True)
    assert name(1184, op="delta_packed") == ("delta_bwd_chunk_kernel", True)
    assert name(296, op="delta_packed", dtype="f32") == ("delta_bwd_chunk_kernel", True)
    assert name(1184, op="delta_packed", dtype="f32") == ("delta_bwd_kernel", False)
