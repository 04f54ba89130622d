"""The host's parallel loops when memory runs out (CPU): the check program is
compiled against csrc/host_parallel.h."""
import subprocess
from pathlib import Path

from mfem_gb300 import build as B


def test_parallel_loops_survive_a_failed_allocation(tmp_path):
    exe = tmp_path / "host_parallel_check"
    src = Path(__file__).resolve().parent / "cpp" / "host_parallel_check.cpp"
    proc = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{B.CSRC}", str(src), "-o", str(exe), "-lpthread"],
                          capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
