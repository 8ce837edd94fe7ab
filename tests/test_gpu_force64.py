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
