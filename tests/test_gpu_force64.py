"""FP64 force kernel, list sort and cell sort at their edges, bit-exact against the oracle: lists that end at, just
before and just after a round of the force kernel and a slot of the sort, CTAs with a partial last atom group, one cell
holding every atom (and a shuffled insertion order), and every soft-repulsion exponent that has its own branch."""
import numpy as np
import pytest

from helpers import make_gpu, make_oracle
from parm_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# a skin of a box length: every other atom is in the list (n - 1 entries), in a single cell
@pytest.mark.parametrize("n", [2, 3, 8, 9, 32, 33, 34, 65, 96, 97, 98, 129, 193, 194, 257])
@pytest.mark.parametrize("kind", [0, 1])
def test_all_pairs_lists(n, kind):
    w = W.small_random(n=n, ndim=3, kind=kind, seed=n, phi=0.4, skin=20.0)
    order = np.random.default_rng(n).permutation(n)
    rank = np.empty(n, dtype=np.uint32)
    rank[order] = np.arange(n)
    g = make_gpu(w, rank=rank)
    o = make_oracle(w, order=[int(i) for i in order])
    g.nlist_update(True)
    o.nl_update(True)
    assert g.numpairs()[0] == n * (n - 1) // 2
    assert np.array_equal(g.pairs(), o.pairs())
    g.set_forces(True)
    o.set_forces(True)
    st, ref = g.get_atoms(), o.get_state()
    assert np.array_equal(st["f"], ref["f"])
    assert np.array_equal(st["a"], ref["a"])


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("exponent,rel", [(2.0, 0.0), (2.5, 1e-13), (3.0, 1e-13)])
def test_repulsion_exponents(ndim, exponent, rel):
    """Exponent 2 takes no power (bit-exact); 5/2 as b sqrt(b) and others by pow within a few ulps a pair."""
    w = W.small_random(n=301, ndim=ndim, kind=1, seed=ndim, phi=0.7, exponent=exponent, skin=0.2)
    g, o = make_gpu(w), make_oracle(w)
    g.nlist_update(True)
    o.nl_update(True)
    g.set_forces(False)
    o.set_forces(False)
    f, ref = g.get_atoms()["f"], o.get_state()["f"]
    assert np.abs(f - ref).max() <= rel * np.abs(ref).max()


@pytest.mark.parametrize("kind,ndim", [(0, 3), (1, 2), (2, 3), (3, 2)])
def test_slots_and_both_sides_agree(kind, ndim):
    """Pair forces kept once per pair, or evaluated for both atoms: the same bits, through rebuilds, on a ragged
    batch whose systems rebuild at different steps (one of them frozen for a while)."""
    ws = [W.small_random(n=n, ndim=ndim, kind=kind, seed=n, phi=0.3, skin=0.3) for n in (5, 61, 130, 311)]
    w = W.Workload("b", ndim, [k.n for k in ws], np.concatenate([k.L for k in ws]), np.concatenate([k.x for k in ws]),
                   np.concatenate([k.v for k in ws]), np.concatenate([k.m for k in ws]), kind,
                   np.concatenate([k.params for k in ws]), 0.3)
    rng = np.random.default_rng(kind)
    rank = np.concatenate([rng.permutation(k.n) for k in ws]).astype(np.uint32)
    out = []
    for keep in (True, False):
        g = make_gpu(w, rank=rank)
        g.debug_pair_slots(keep)
        g.nlist_update(False)
        g.set_forces(True)
        g.damped(1e-4, 5.0, 20)
        g.set_active([1, 1, 0, 1])
        g.damped(1e-4, 5.0, 40)
        g.set_active([1, 1, 1, 1])
        g.set_capacity(g.capacity() + 24)   # lists re-pitched between rebuilds
        g.damped(1e-4, 5.0, 40)
        g.nlist_update(True)
        g.damped(1e-4, 5.0, 4)
        out.append((g.get_atoms(), g.which()))
    for k in ("x", "v", "a", "f"):
        assert np.array_equal(out[0][0][k], out[1][0][k])
    assert np.array_equal(out[0][1], out[1][1]) and out[0][1].min() > 1


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 34, 64, 65, 66, 97, 130])
def test_cluster_in_a_large_box(n, ndim):
    """The kernel for short lists (chosen by the mean list and the atom count) on lists that are not: every atom of a
    small cluster in each list, one round of the kernel and more; a second system of lone atoms makes up the count."""
    w = W.small_random(n=n, ndim=ndim, kind=1, seed=n, phi=0.6, skin=30.0)
    w.L[:] = 400.0
    o = make_oracle(w)
    lone = 8192
    gap = 40.0   # beyond every list
    k = 21 if ndim == 3 else 91
    x = (np.stack(np.meshgrid(*[np.arange(k)] * ndim, indexing="ij"), -1).reshape(-1, ndim)[:lone] + 0.5) * gap
    g = make_gpu(W.Workload("c", ndim, [n, lone], np.array([[400.0] * ndim, [k * gap] * ndim]),
                            np.concatenate([w.x, x]), np.zeros((n + lone, ndim)),
                            np.concatenate([w.m, np.ones(lone)]), 1,
                            np.concatenate([w.params, np.tile(w.params[:1], (lone, 1))]), 30.0))
    g.set_capacity(n)
    g.nlist_update(True)
    o.nl_update(True)
    assert g.numpairs()[0] == n * (n - 1) // 2
    g.set_forces(True)
    o.set_forces(True)
    st, ref = g.get_atoms(), o.get_state()
    assert np.array_equal(st["f"][:n], ref["f"]) and not st["f"][n:].any()
    assert np.array_equal(st["a"][:n], ref["a"])


def test_slots_of_tiny_systems():
    """Eight lists of a CTA out of up to eight systems, of which some rebuild and others do not."""
    sizes = [1, 2, 3, 1, 5, 8, 9, 1, 1, 1, 7, 16, 17, 2, 30, 1, 4, 6]
    ws = [W.small_random(n=n, ndim=3, kind=0, seed=k, phi=0.2, skin=0.3) for k, n in enumerate(sizes)]
    w = W.Workload("t", 3, sizes, np.concatenate([k.L for k in ws]), np.concatenate([k.x for k in ws]),
                   np.concatenate([k.v for k in ws]), np.concatenate([k.m for k in ws]), 0,
                   np.concatenate([k.params for k in ws]), 0.3)
    out = []
    for keep in (True, False):
        g = make_gpu(w)
        g.debug_pair_slots(keep)
        g.nlist_update(False)
        g.set_forces(True)
        for q in range(3):
            g.set_active([(k + q) % 3 != 0 for k in range(len(sizes))])
            g.damped(1e-4, 5.0, 30)
        out.append((g.get_atoms(), g.which()))
    for k in ("x", "v", "a", "f"):
        assert np.array_equal(out[0][0][k], out[1][0][k])
    assert np.array_equal(out[0][1], out[1][1]) and out[0][1].max() > 1


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("n", [2, 16, 17, 18, 33, 130, 240])
def test_cluster_among_many_atoms(ndim, n):
    """The kernel for many atoms on lists of one round and more, with more survivors than it holds at once."""
    w = W.small_random(n=n, ndim=ndim, kind=1, seed=n, phi=3.0, skin=30.0)
    w.L[:] = 400.0
    o = make_oracle(w)
    gap = 40.0   # beyond every list
    k = 42 if ndim == 3 else 271
    x = (np.stack(np.meshgrid(*[np.arange(k)] * ndim, indexing="ij"), -1).reshape(-1, ndim) + 0.5) * gap
    lone = len(x)
    assert lone > 152 * 15 * 32
    g = make_gpu(W.Workload("c", ndim, [n, lone], np.array([[400.0] * ndim, [k * gap] * ndim]),
                            np.concatenate([w.x, x]), np.zeros((n + lone, ndim)),
                            np.concatenate([w.m, np.ones(lone)]), 1,
                            np.concatenate([w.params, np.tile(w.params[:1], (lone, 1))]), 30.0))
    g.set_capacity(n)
    g.nlist_update(True)
    o.nl_update(True)
    assert g.numpairs()[0] == n * (n - 1) // 2
    g.set_forces(True)
    o.set_forces(True)
    st, ref = g.get_atoms(), o.get_state()
    assert np.array_equal(st["f"][:n], ref["f"]) and not st["f"][n:].any()
    assert np.array_equal(st["a"][:n], ref["a"])


@pytest.mark.parametrize("kind,ndim,expo,skin", [(1, 2, 2.0, 0.2), (1, 3, 2.5, 0.2), (2, 3, 2.0, 0.2), (2, 2, 2.0, 1.5),
                                                 (1, 2, 3.0, 0.1)])
def test_many_atoms_and_slots_agree(kind, ndim, expo, skin):
    """The kernel for many atoms against pair forces kept once per pair: the same bits on ragged batches, one frozen."""
    ws = [W.small_random(n=n, ndim=ndim, kind=kind, seed=n, phi=0.7, skin=skin, exponent=expo) for n in (70001, 3001, 61)]
    w = W.Workload("b", ndim, [k.n for k in ws], np.concatenate([k.L for k in ws]), np.concatenate([k.x for k in ws]),
                   np.concatenate([k.v for k in ws]), np.concatenate([k.m for k in ws]), kind,
                   np.concatenate([k.params for k in ws]), skin)
    assert w.n > 152 * 15 * 32
    dt = 1e-5 if kind == 1 else 1e-14   # (random positions: WCA forces of 1e30)
    out = []
    for keep in (True, False):
        g = make_gpu(w)
        g.debug_pair_slots(keep)
        g.nlist_update(False)
        g.set_forces(True)
        g.damped(dt, 5.0, 5)
        g.set_active([1, 0, 1])
        g.damped(dt, 5.0, 10)
        out.append(g.get_atoms())
    for k in ("x", "v", "a", "f"):
        assert np.array_equal(out[0][k], out[1][k])
