"""The force kernels' quotient from a shared reciprocal (parm_gb300/csrc/fpbits.cuh) equals the division, bit for bit
(tests/programs/quotient_check.cpp)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_quotient_by_reciprocal_is_the_quotient(tmp_path):
    exe = tmp_path / "quotient_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'parm_gb300' / 'csrc'}",
                        str(ROOT / "tests" / "programs" / "quotient_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
