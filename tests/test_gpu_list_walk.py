"""GPU: the plain walks by interaction lists (k_walk_list64) at the counts where
they can go wrong -- ragged buckets, lists that do not fit and go back to the walks
by warp, both sides of the target count that selects them -- against the oracle.  Bit
equality, counters included."""
import numpy as np
import pytest

import pepc_b200 as P
from oracle import oracle as O
from tests.datasets import cube, plummer

pytestmark = pytest.mark.gpu
KEYS = ("ex", "ey", "ez", "pot", "work")


def both(x, y, z, q, walk, nt=None, shift=0.0, **kw):
    """Fields of the grown particles, or of the first nt of them moved by shift."""
    tc = P.TreeCode(walk=walk, **kw)
    orc = O.Oracle(walk=0 if walk == P.WALK_PER_TARGET else 1, num_threads=8, **kw)
    g, go = tc.pepc_grow_tree(x, y, z, q), orc.grow_tree(x, y, z, q)
    t = [a[:nt] + shift for a in (g.x, g.y, g.z)]
    keys = {} if nt is not None and walk == P.WALK_PER_TARGET else dict(keys=g.key)
    r, ro = tc.pepc_traverse_tree(*t, **keys), orc.traverse_tree(*t, **keys)
    for k in KEYS:
        assert np.array_equal(r[k], ro[k]), k
    c = orc.counters()
    st = tc.stats()
    assert st["interactions"] == c["interactions"]
    tc.close()
    orc.close()
    return st


@pytest.mark.parametrize("walk", [P.WALK_PER_TARGET, P.WALK_PER_TILE])
@pytest.mark.parametrize("n", [2, 31, 33, 500, 4099, 20011, 65536, 65537])
def test_self_fields(gpu, n, walk):
    both(*cube(n, 71, charges="gauss"), walk, theta2=0.36, eps2=1e-6)


@pytest.mark.parametrize("walk", [P.WALK_PER_TARGET, P.WALK_PER_TILE])
def test_lists_that_do_not_fit(gpu, walk):
    # a clustered tree, theta 0.36: some unions of 32 lists are longer than a list, the
    # others are not
    both(*plummer(40000, 72), walk, theta2=0.13, eps2=1e-6)


# buckets of 8, 16 and 32 targets anywhere on a clustered tree, theta 0.36: unions that fit,
# that fit in parts, and that do not fit with four targets either
@pytest.mark.parametrize("nt", [3, 1003, 4735, 20011])
@pytest.mark.parametrize("n", [40000, 200000])
def test_scattered_targets(gpu, n, nt):
    kw = dict(theta2=0.13, eps2=1e-6)
    x, y, z, q = plummer(n, 72)
    tc, orc = P.TreeCode(**kw), O.Oracle(num_threads=8, **kw)
    tc.pepc_grow_tree(x, y, z, q)
    orc.grow_tree(x, y, z, q)
    t = np.random.default_rng(73).permutation(len(x))[:nt]
    a, b = tc.pepc_traverse_tree(x[t], y[t], z[t]), orc.traverse_tree(x[t], y[t], z[t])
    for k in KEYS:
        assert np.array_equal(a[k], b[k]), k
    st, c = tc.stats(), orc.counters()
    assert st["interactions"] == c["interactions"]
    tc.close()
    orc.close()


@pytest.mark.parametrize("nt", [1, 32, 33, 24576, 24577])
def test_target_counts(gpu, nt):
    # targets beside the particles, without keys, on both sides of the line at 24,576
    both(*cube(66000, 74), P.WALK_PER_TARGET, nt=nt, shift=1e-3, theta2=0.5, eps2=1e-4)


@pytest.mark.parametrize("mac", [1, 2])
def test_other_opening_criteria(gpu, mac):
    # Bmax, and no acceptance at all (every list holds every leaf)
    both(*cube(3000, 75), P.WALK_PER_TARGET, theta2=0.36, eps2=1e-4, mac_select=mac)


def test_results_accumulate(gpu):
    x, y, z, q = cube(700, 76)
    tc, orc = P.TreeCode(theta2=0.36), O.Oracle(theta2=0.36, num_threads=8)
    g, go = tc.pepc_grow_tree(x, y, z, q), orc.grow_tree(x, y, z, q)
    e = [np.linspace(-1, 1, 700) for _ in range(3)]
    pot, work = np.full(700, 0.25), np.full(700, 0.1)
    base = tc.pepc_traverse_tree(g.x, g.y, g.z)
    r = tc.pepc_traverse_tree(g.x, g.y, g.z, e=e, pot=pot, work=work)
    # the same terms, added one by one to the given start
    assert np.allclose(r["ex"], base["ex"] + e[0], rtol=1e-12, atol=1e-12)
    w = np.full(700, 0.1)
    for i in range(700):
        for _ in range(int(base["work"][i])):
            w[i] += 1.0
    assert np.array_equal(r["work"], w)
