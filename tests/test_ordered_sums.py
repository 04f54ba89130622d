"""The resident PCG's ordered sums on the host (CPU): the check program is
compiled against csrc/partition.cpp and runs without a GPU."""
import subprocess
from pathlib import Path

from mfem_gb300 import build as B


def test_ordered_sums_reach_every_component(tmp_path):
    exe = tmp_path / "ordered_sums_check"
    src = Path(__file__).resolve().parent / "cpp" / "ordered_sums_check.cpp"
    proc = subprocess.run([B.nvcc_path(), "-x", "cu", "-std=c++17", "-O1", f"-I{B.INCLUDE}", f"-I{B.CSRC}", str(src),
                           str(B.CSRC / "partition.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
