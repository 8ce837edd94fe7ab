"""Radius and angle of the Langevin normals at chosen 53-bit variates v, against quadruple precision: the ends of the range,
both sides of every interval of the tables in every binade (the split at sqrt 2 and the interval next to 1 among them),
and the angle's ties.  In units of 2^-53: the radius within 2 of itself (one for the logarithm's sum and its table entry,
halved by the root, one for the root), cosine and sine within 1.5 (half each for the table, its product and the sum)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent
TOP = 1 << 53


@pytest.fixture(scope="module")
def noise():
    from parm_gb300.build import CSRC, nvcc
    if np.finfo(np.longdouble).eps > 1e-19:
        pytest.skip("long double is no wider than double here")
    out = HERE / "_build" / "libnoise_words.so"
    out.parent.mkdir(exist_ok=True)
    subprocess.run([nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "--expt-relaxed-constexpr", f"-I{CSRC}", "-Xcompiler", "-fPIC", "-shared",
                    str(HERE / "csrc" / "noise_words.cu"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))

    def call(v):
        v = np.ascontiguousarray(sorted({int(k) for k in v if 0 <= k < TOP}), dtype=np.uint64)
        res = np.zeros((len(v), 3))
        assert lib.noise_words(v.ctypes.data_as(C.POINTER(C.c_uint64)), res.ctypes.data_as(C.POINTER(C.c_double)),
                               C.c_uint32(len(v))) == 0
        return v, res
    return call


def _near(points, width=3):
    return [int(p) + d for p in points for d in range(-width, width + 1)]


def _check_radius(noise, words):
    v, res = noise(words)
    u = ((v.astype(np.float64) + 0.5) * 2.0 ** -53)       # as FP64 rounds it: 1 for the last one
    r = np.sqrt(np.longdouble(-2) * np.log(u.astype(np.longdouble)))
    one = u == 1.0
    assert not res[one, 0].any()
    err = np.abs(res[~one, 0] - r[~one]) / r[~one]
    assert err.max() <= 2 * 2.0 ** -53, v[~one][err.argmax()]


def test_radius_at_the_ends(noise):
    _check_radius(noise, list(range(4096)) + list(range(TOP - 4096, TOP)) + _near([TOP >> 1, TOP >> 2, 3 * (TOP >> 2)], 64))


def test_radius_at_the_table_s_intervals(noise):
    # 2 v + 1 next to (1 + k / 128) 2^e
    _check_radius(noise, _near([(128 + k) * 2 ** e // 256 for e in range(54) for k in range(129)]))


def test_angle_at_ties_and_ends(noise):
    # 2 v + 1 next to k 2^45 (table angles) and (k + 1/2) 2^45 (ties between them)
    v, res = noise(_near([k * 2 ** 43 for k in range(1025)]) + list(range(64)) + list(range(TOP - 64, TOP)))
    L = np.longdouble
    th = (v.astype(L) + L(0.5)) * L(2) ** -53 * (L(4) * np.arccos(L(0)))
    assert np.abs(res[:, 1] - np.cos(th)).max() <= 1.5 * 2.0 ** -53
    assert np.abs(res[:, 2] - np.sin(th)).max() <= 1.5 * 2.0 ** -53
