"""Host check of the work buffers that outlive a call (no GPU): what a failed allocation leaves behind."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_buffers_after_a_failed_allocation(tmp_path):
    exe = tmp_path / "buf_host_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(exe), str(ROOT / "tests" / "buf_host_check.cpp")], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    assert p.stdout.strip() == "errors: 0"
