"""Host check of the counting sort's place checks (no GPU): keys that change while they are sorted are reported."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_keys_that_change_are_reported(tmp_path):
    exe = tmp_path / "sort_host_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", str(exe), str(ROOT / "tests" / "sort_host_check.cpp")], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    assert p.stdout.strip() == "errors: 0"
