"""Which commands of a replayed Tile program share a launch, on the host: in any order the commands that join leave memory as
they do one by one."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_what_joins_does_not_depend_on_its_order(tmp_path):
    program = tmp_path / "replay_rules_check"
    subprocess.run(["g++", "-std=c++17", "-O1", str(ROOT / "tests/host_cpp/replay_rules_check.cpp"), "-o", str(program)], check=True,
                   capture_output=True, text=True, timeout=300)
    result = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and "PASS" in result.stdout, result.stdout + result.stderr
