"""What the assembler reports for kernels whose speed hangs on it."""
import re
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_formal_gemm_forms_keep_their_registers(tmp_path):
    # 64 registers (four blocks of 256 threads to an SM) hold every form; a shifted copy of its arguments made three of them spill
    from vibe_compiler_b200.build import NVCC_FLAGS
    result = subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", *NVCC_FLAGS, "-Xptxas", "-v", "-c",
                             str(ROOT / "vibe_compiler_b200/csrc/gemm_formal.cu"), "-o", str(tmp_path / "gemm_formal.o")],
                            check=True, capture_output=True, text=True, timeout=600)
    found = re.findall(r"Compiling entry function '\S*gemm_formal_\w+_kernel.*?(\d+) bytes stack frame, (\d+) bytes spill stores", result.stderr, re.S)
    assert len(found) >= 4 and all(entry == ("0", "0") for entry in found), found
