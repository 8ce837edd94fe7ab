"""Calls between set_interaction and the next list build, on the lists there are: none on a new handle, else those of the
last build (the pair kernels and the evaluation must not read what only a build writes: the tables of the cell blocks on a
new grid, the pair slots of new ranks)."""
import numpy as np
import pytest

from helpers import make_gpu
from parm_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _all(g):
    g.set_forces(True)
    return [g.energy(), g.virial(), g.stress(), g.contacts(), g.overlaps(), g.numpairs(), g.get_atoms()["f"]]


def _same(got, ref):
    for a, b in zip(got[3:6], ref[3:6]):
        assert np.array_equal(a, b)
    scales = [np.abs(ref[0]), np.abs(ref[1]), np.abs(ref[1])[:, None, None]]
    for a, b, s in zip(got[:3], ref[:3], scales):
        assert np.all(np.abs(a - b) <= 1e-6 * s)
    assert np.abs(got[6] - ref[6]).max() <= 1e-5 * np.abs(ref[6]).max()


def _work(kind=1, n=2000, skin=0.2):
    return W.small_random(n=n, ndim=3, kind=kind, seed=kind, phi=0.5, skin=skin)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_new_handle(precision):
    w = _work()
    g = make_gpu(w, precision=precision)
    for a in _all(g):
        assert not np.any(a)
    g.nlist_update(False)
    h = make_gpu(w, precision=precision)
    h.nlist_update(False)
    a, b = _all(g), _all(h)
    assert a[5][0] > 1000
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    assert np.array_equal(g.which(), h.which())


@pytest.mark.parametrize("slots", [0, 1])
def test_old_lists_on_a_new_grid(slots):
    """A longer skin: other cells, and until the next build the old pairs."""
    w, wide = _work(), _work(skin=0.9)
    g, ref = make_gpu(w, precision="mixed"), make_gpu(w, precision="mixed")
    ref.set_threads_per_atom(101)
    for h in (g, ref):
        h.nlist_update(False)
        h.set_interaction(wide.kind, wide.params, wide.skin)
    assert g.threads_per_atom() == 200
    got, want = _all(g), _all(ref)
    assert want[5][0] > 1000
    _same(got, want)
    if slots:                       # the lists also survive a change of their kernel and of their capacity
        g.set_capacity(g.capacity() + 16)
        g.set_threads_per_atom(101)
        _same(_all(g), want)
        g.set_threads_per_atom(200)
        _same(_all(g), want)
    for h in (g, ref):
        h.nlist_update(False)
        assert h.which()[0] == 2
    _same(_all(g), _all(ref))


def test_autotune_of_a_new_handle():
    w = _work()
    g, h = make_gpu(w, precision="mixed"), make_gpu(w, precision="mixed")
    g.autotune()
    h.nlist_update(False)
    assert np.array_equal(g.pairs(), h.pairs())
    g.nlist_update(False)
    assert g.which()[0] == 1


@pytest.mark.parametrize("grown", [False, True])
def test_pair_slots_after_new_ranks(grown):
    """Half of the atoms leave the list, positions move, forces are asked for before the next build."""
    w = W.small_random(n=700, ndim=3, kind=0, seed=3, phi=0.3, skin=0.3)
    rank = np.random.default_rng(1).permutation(w.n).astype(np.uint32)
    left = np.where(np.arange(w.n) % 2 == 0, rank, np.uint32(0xFFFFFFFF)).astype(np.uint32)
    out = []
    for keep in (0, 1):
        g = make_gpu(w, rank=rank)
        g.debug_pair_slots(keep)
        g.nlist_update(False)
        g.set_forces(True)
        g.set_atoms(x=w.x * 1.001)
        g.set_interaction(w.kind, w.params, w.skin, rank=left)
        if grown:
            g.set_capacity(g.capacity() + 40)
        g.set_forces(True)
        first = g.get_atoms()["f"]
        g.verlet(1e-5, 3)
        out.append((first, g.get_atoms()["f"], g.which()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("boxed", [False, True])
def test_minimiser_before_the_first_build(boxed):
    w = W.small_random(n=700, ndim=3, kind=1, seed=3, phi=0.6, skin=0.3)
    out = []
    for keep in (0, 1):
        g = make_gpu(w)
        g.debug_pair_slots(keep)
        g.nlcg_init([0.1, 1e-4, 10.0, 1000.0, 10.0, 1e-4, 0.0, 0.0, 0.0, 0.0, 0.0], boxed=boxed)
        g.nlcg_reset()
        g.nlcg_timestep(3)
        out.append((g.get_atoms()["x"], g.get_atoms()["f"], g.which()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_old_lists_under_a_law_without_cell_blocks():
    """The attractive LJ on the grid of the LJ lists: the per-atom kernels take over, on the same pairs."""
    w = _work(kind=0)
    g, ref = make_gpu(w, precision="mixed"), make_gpu(w, precision="mixed")
    ref.set_threads_per_atom(101)
    for h in (g, ref):
        h.nlist_update(False)
        h.set_interaction(3, w.params, w.skin)
    got, want = _all(g), _all(ref)
    assert want[5][0] > 1000
    _same(got, want)
