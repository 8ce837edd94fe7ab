"""The force kernels' b^(3/2) against exact arithmetic: |result - b^(3/2)| <= (1/2 + 2^-40) ulp, that is
(2 r - u)^2 <= 4 b^3 <= (2 r + u)^2 in rationals, u one ulp (tests/programs/three_halves.cpp)."""
import struct
import subprocess
from fractions import Fraction
from math import ulp
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_three_halves_is_rounded_once(tmp_path):
    exe = tmp_path / "three_halves"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'parm_gb300' / 'csrc'}",
                        str(ROOT / "tests" / "programs" / "three_halves.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0
    n = 0
    for line in r.stdout.split("\n"):
        if not line:
            continue
        b, y = (struct.unpack("<d", struct.pack("<Q", int(h, 16)))[0] for h in line.split())
        u = Fraction(ulp(y)) * (1 + Fraction(1, 2 ** 39))
        assert (2 * Fraction(y) - u) ** 2 <= 4 * Fraction(b) ** 3 <= (2 * Fraction(y) + u) ** 2 or y == b == 0.0, (b, y)
        n += 1
    assert n > 60000
