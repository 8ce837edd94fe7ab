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
