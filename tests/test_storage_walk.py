"""The walk of the elementwise and convert commands over physical storage, compared on the host with the row-major-to-physical
map: every layout, ranks 1 to 5, ragged and empty shapes, all pairs of formats, extents whose products pass 32 bits."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_walk_visits_the_elements_of_every_layout(tmp_path):
    program = tmp_path / "storage_walk_check"
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    str(ROOT / "tests/host_cpp/storage_walk_check.cu"), str(ROOT / "vibe_compiler_b200/csrc/layout.cu"), "-o", str(program)],
                   check=True, capture_output=True, text=True, timeout=600)
    result = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and "PASS" in result.stdout, result.stdout + result.stderr
