"""Evaluation on the cell-block lists against the per-atom kernels on the same lists: every law, uniform and per-atom
parameters, 2D and 3D, ragged batches, whole neighbourhoods in shared memory or (stage capacity 32) nearly none of them.
Counts equal; sums of FP32 pair terms whose displacements round alike but for periodic images: 1e-6 of the sum of
magnitudes is a hundred times the FP32 rounding of such sums."""
import numpy as np
import pytest

from helpers import make_gpu
from parm_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,ndim,bidisperse,expo", [(0, 3, False, 2.0), (0, 3, True, 2.0), (0, 2, True, 2.0),
                                                       (1, 2, True, 2.0), (1, 3, True, 2.5), (1, 3, False, 3.0),
                                                       (2, 3, True, 2.0), (2, 2, False, 2.0)])
@pytest.mark.parametrize("cap", [0, 32])
def test_staged_evaluation_matches_gather(kind, ndim, bidisperse, expo, cap):
    ws = [W.small_random(n=n, ndim=ndim, kind=kind, seed=n, phi=0.5, skin=0.2, bidisperse=bidisperse, exponent=expo)
          for n in (1500, 2111)]
    w = W.Workload("b", ndim, [k.n for k in ws], np.concatenate([k.L for k in ws]), np.concatenate([k.x for k in ws]),
                   np.concatenate([k.v for k in ws]), np.concatenate([k.m for k in ws]), kind,
                   np.concatenate([k.params for k in ws]), 0.2)
    rank = np.concatenate([np.random.default_rng(n).permutation(k.n) for n, k in enumerate(ws)]).astype(np.uint32)
    g = make_gpu(w, precision="mixed", rank=rank)
    g.nlist_update(True)
    assert g.threads_per_atom() == 200
    if cap:
        g.debug_stage_cap(cap)
    got = [g.energy(), g.virial(), g.stress(), g.contacts(), g.overlaps(), g.numpairs()]
    g.debug_stage_cap(0)
    g.set_threads_per_atom(101)
    ref = [g.energy(), g.virial(), g.stress(), g.contacts(), g.overlaps(), g.numpairs()]
    for a, b in zip(got[3:], ref[3:]):
        assert np.array_equal(a, b)
    assert ref[5].min() > 100
    for a, b, scale in zip(got[:3], ref[:3], (np.abs(ref[0]), np.abs(ref[1]), np.abs(ref[1])[:, None, None])):
        assert np.all(np.abs(a - b) <= 1e-6 * scale)


def _both(w):
    """Energy, virial, contacts, overlaps on the cell-block lists and by the per-atom kernels."""
    g = make_gpu(w, precision="mixed")
    g.nlist_update(True)
    assert g.threads_per_atom() == 200
    got = [g.energy(), g.virial(), g.contacts(), g.overlaps()]
    g.set_threads_per_atom(101)
    return got, [g.energy(), g.virial(), g.contacts(), g.overlaps()]


@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("bidisperse", [False, True])
@pytest.mark.parametrize("apart", [0.0, 1e-8, 1e-7, 3e-7])
def test_atoms_on_top_of_each_other(kind, bidisperse, apart):
    """(r / sigma)^6 below the FP32 range: the energy is +inf, and the pair a contact and an overlap."""
    w = W.small_random(n=1500, ndim=3, kind=kind, seed=4, phi=0.4, skin=0.2, bidisperse=bidisperse)
    w.x[7] = w.x[1400] = np.floor(w.x[7] * 8) / 8
    w.x[7, 1] += apart
    got, ref = _both(w)
    assert np.isposinf(ref[0][0]) and np.isposinf(got[0][0])
    assert np.array_equal(got[2], ref[2]) and np.array_equal(got[3], ref[3])


@pytest.mark.parametrize("kind,expo,bidisperse", [(0, 2.0, False), (0, 2.0, True), (2, 2.0, False), (2, 2.0, True),
                                                  (1, 2.0, True), (1, 2.5, True), (1, 3.0, True)])
def test_the_same_pair_terms(kind, expo, bidisperse):
    """Positions in 256ths and a box in eighths: every displacement and squared distance is exact in FP32, so the pair
    terms are those of the per-atom kernels and the sums differ by the order of their FP64 additions only."""
    k = 14
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(g)
    x = g + 0.5 + np.random.default_rng(5).integers(-40, 41, size=g.shape) / 256.0
    sig = np.where(np.arange(n) % 3 == 0, 1.25, 1.0) if bidisperse else np.ones(n)
    third = {0: W.LJ_SIGCUT, 1: expo, 2: 0.0}[kind]
    w = W.Workload("e", 3, [n], np.full((1, 3), float(k)), x, np.zeros((n, 3)), np.ones(n), kind,
                   np.stack([np.ones(n), sig, np.full(n, third)], 1), 0.2)
    got, ref = _both(w)
    for a, b in zip(got[:2], ref[:2]):
        assert abs(a[0] - b[0]) <= 1e-12 * max(abs(b[0]), n)
    assert np.array_equal(got[2], ref[2]) and np.array_equal(got[3], ref[3])
