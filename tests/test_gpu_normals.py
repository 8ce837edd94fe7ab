"""The Langevin normals against quadruple precision: radius sqrt(-2 log u) and angle 2 pi u of the same Philox words, at
counters drawn at random and at words whose uniforms lie at the ends of their range (the bit patterns themselves are
covered by the Philox tests).  The bound is 4 units of 2^-53 of the radius: one for the logarithm's sum, half for each of
root, table, angle and product."""
import numpy as np
import pytest

from philox_py import philox_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,step,n", [(0, 1, 60000), (99, 123456789012, 60000)])
def test_normals_to_four_units(seed, step, n):
    from oracle.oracle import splitmix64
    from parm_gb300.system import debug_normals
    if np.finfo(np.longdouble).eps > 1e-19:
        pytest.skip("long double is no wider than double here")
    got = debug_normals(seed, 2, step, n)
    key = splitmix64(seed + 2)
    L = np.longdouble
    pi = L(2) * np.arccos(L(0))
    for blk in range(3):
        rows = np.zeros((n, 6), dtype=np.uint32)
        rows[:, 0] = np.arange(n)
        rows[:, 1], rows[:, 2], rows[:, 3] = step & 0xFFFFFFFF, step >> 32, blk
        rows[:, 4], rows[:, 5] = key & 0xFFFFFFFF, key >> 32
        w = philox_rows(rows).astype(np.uint64)
        v = [(w[:, k] >> np.uint64(5)) << np.uint64(26) | (w[:, k + 1] >> np.uint64(6)) for k in (0, 2)]
        u1 = ((v[0].astype(np.float64) + 0.5) * 2.0 ** -53).astype(L)   # the variate as FP64 rounds it
        r = np.sqrt(L(-2) * np.log(u1))
        th = L(2) * pi * ((v[1].astype(L) + L(0.5)) * L(2) ** -53)
        for k, f in ((0, np.cos), (1, np.sin)):
            err = np.abs(got[:, 2 * blk + k].astype(L) - r * f(th)) / r
            assert err.max() <= 4 * 2.0 ** -53
