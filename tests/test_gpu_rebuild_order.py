"""The permutation of a rebuild where it has large groups to move: atoms outside the neighbour list, and cells of
hundreds of atoms, each with a time that a single warp for the group would miss by far."""
import time

import numpy as np
import pytest

from helpers import make_gpu, make_oracle
from parm_gb300 import workloads as W
from parm_gb300.capi import NOT_MEMBER

pytestmark = pytest.mark.gpu


def _fastest_rebuild(g, times=5):
    best = 1e9
    for _ in range(times):
        t = time.perf_counter()
        g.nlist_update(True)
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("masses", [False, True])
def test_few_members_among_many_atoms(ndim, masses):
    """Two systems with every seventh and every second atom in the list: the members move as they do alone, bit for bit,
    the others on their own."""
    ws = [W.small_random(n=n, ndim=ndim, kind=1, seed=n, phi=2.0, skin=0.2) for n in (3001, 500)]
    m = np.concatenate([k.m for k in ws]) if masses else np.full(3501, 2.0)
    w = W.Workload("nm", ndim, [k.n for k in ws], np.concatenate([k.L for k in ws]), np.concatenate([k.x for k in ws]),
                   np.concatenate([k.v for k in ws]), m, 1, np.concatenate([k.params for k in ws]), 0.2)
    member = np.concatenate([np.arange(3001) % 7 == 3, np.arange(500) % 2 == 1])
    rng = np.random.default_rng(ndim)
    rank = np.full(w.n, NOT_MEMBER, dtype=np.uint32)
    parts = np.split(np.arange(w.n), [3001])
    for p in parts:
        k = p[member[p]]
        rank[k] = rng.permutation(len(k))
    g = make_gpu(w, rank=rank)
    alone = W.Workload("m", ndim, [int(member[p].sum()) for p in parts], w.L, w.x[member], w.v[member], m[member], 1,
                       w.params[member], 0.2)
    h = make_gpu(alone, rank=rank[member])
    for s in (g, h):
        s.nlist_update(False)
        s.set_forces(True)
        s.verlet(0.01, 60)
    assert g.which().min() > 2 and np.array_equal(g.which(), h.which())
    a, b = g.get_atoms(), h.get_atoms()
    for k in ("x", "v", "a", "f"):
        assert np.array_equal(a[k][member], b[k])
    assert not a["f"][~member].any()
    assert np.array_equal(a["v"][~member], w.v[~member]) and np.array_equal(a["m"], m)
    x = w.x[~member] + 60 * 0.01 * w.v[~member]
    assert np.abs(a["x"][~member] - x).max() < 1e-11


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rebuild_time_with_few_members(precision):
    """400,000 atoms, 1000 of them in the list, against all of them in it: less to do, so not longer (a warp for all the
    others takes tens of times as long)."""
    n = 400_000
    w = W.soft_disks(n=n, phi=0.5)
    rank = np.full(n, NOT_MEMBER, dtype=np.uint32)
    rank[:1000] = np.arange(1000)
    t = [_fastest_rebuild(make_gpu(w, precision=precision, rank=r)) for r in (rank, None)]
    print("few / all members: %.0f / %.0f us" % (1e6 * t[0], 1e6 * t[1]))
    assert t[0] < 2.0 * t[1]


def test_one_cell_of_hundreds_in_order():
    """700 atoms in a single cell in a shuffled list order: lists and forces as the oracle's, bit for bit."""
    w = W.small_random(n=700, ndim=3, kind=0, seed=8, phi=0.62, skin=0.4)
    order = np.random.default_rng(8).permutation(w.n)
    rank = np.empty(w.n, dtype=np.uint32)
    rank[order] = np.arange(w.n)
    g, o = make_gpu(w, rank=rank), make_oracle(w, order=[int(i) for i in order])
    g.nlist_update(True)
    o.nl_update(True)
    assert np.array_equal(g.pairs(), o.pairs())
    g.set_forces(True)
    o.set_forces(True)
    assert np.array_equal(g.get_atoms()["f"], o.get_state()["f"])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ndim,n,side", [(2, 9001, 1.0), (2, 30011, 0.5), (2, 60007, 1.1), (3, 20011, 0.75),
                                         (3, 50021, 1.4)])
def test_sparse_cells(precision, ndim, n, side):
    """One to seven atoms a cell in the mean: no atom is lost or doubled, the pairs are those of a tree."""
    cKDTree = pytest.importorskip("scipy.spatial").cKDTree
    rl = 1.3
    L = side * n ** (1.0 / ndim)
    x = np.random.default_rng(n).uniform(0, L, size=(n, ndim))
    m = 1.0 + np.arange(n) % 3
    w = W.Workload("s", ndim, [n], np.full((1, ndim), L), x, x * 0.5, m, 1, np.tile([1.0, 1.0, 2.0], (n, 1)), rl - 1.0)
    g = make_gpu(w, precision=precision)
    for _ in range(3):
        g.nlist_update(True)
    st = g.get_atoms()
    assert np.array_equal(st["x"], x) and np.array_equal(st["v"], w.v) and np.array_equal(st["m"], m)
    tree = cKDTree(np.mod(x, L), boxsize=L)
    assert int(g.numpairs()[0]) == len(tree.query_pairs(rl, output_type="ndarray"))


@pytest.mark.parametrize("n,side", [(9001, 1.0), (30011, 1.2), (50021, 1.4)])
def test_dense_cells_among_sparse_ones(n, side):
    """Four cells of some 70 atoms in a batch of cells of one or two: sixteen, eight and four lanes a group, three groups
    a cell.  The pairs of both systems are those of a tree, and no atom is lost."""
    cKDTree = pytest.importorskip("scipy.spatial").cKDTree
    rng, rl = np.random.default_rng(n), 1.29
    sizes, L = [280, n], [2.59, side * n ** 0.5]
    x = np.concatenate([rng.uniform(0, b, size=(k, 2)) for k, b in zip(sizes, L)])
    w = W.Workload("d", 2, sizes, np.repeat(np.array(L)[:, None], 2, axis=1), x, x * 0.5, 1.0 + np.arange(len(x)) % 3, 1,
                   np.tile([1.0, 1.0, 2.0], (len(x), 1)), rl - 1.0)
    g = make_gpu(w)
    for _ in range(3):
        g.nlist_update(True)
    st = g.get_atoms()
    assert np.array_equal(st["x"], x) and np.array_equal(st["v"], w.v) and np.array_equal(st["m"], w.m)
    trees = [cKDTree(p, boxsize=b) for p, b in zip(np.split(x, [280]), L)]
    assert [int(k) for k in g.numpairs()] == [len(t.query_pairs(rl, output_type="ndarray")) for t in trees]
