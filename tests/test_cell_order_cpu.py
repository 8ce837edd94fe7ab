"""The order of the cells in tiles along y is a numbering of the grid and cell_coords its inverse
(tests/programs/cell_order_check.cu, compiled for the host)."""
import subprocess
from pathlib import Path

from parm_gb300.build import nvcc

ROOT = Path(__file__).resolve().parent.parent


def test_cell_order_is_a_numbering(tmp_path):
    exe = tmp_path / "cell_order_check"
    r = subprocess.run([nvcc(), "-std=c++17", "-O2", f"-I{ROOT / 'parm_gb300' / 'csrc'}",
                        str(ROOT / "tests" / "programs" / "cell_order_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
