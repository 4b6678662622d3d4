"""How tensor-core GEMMs are cut over the SMs, on the host: rings and accumulators fit, every tile has a CTA, and where SMs are
kept for a sum that runs beside a layer's kernels no more CTAs than the others are launched."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_cuts_fit_and_leave_the_kept_sms_free(tmp_path):
    program = tmp_path / "gemm_plan_check"
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    str(ROOT / "tests/host_cpp/gemm_plan_check.cu"), str(ROOT / "vibe_compiler_b200/csrc/layout.cu"), "-o", str(program)],
                   check=True, capture_output=True, text=True, timeout=600)
    result = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and "PASS" in result.stdout, result.stdout + result.stderr
