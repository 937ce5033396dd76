"""GPU: the grow's kernels at the sizes where their choice or their work split
changes: the one-launch sort's tiles (1,024, 2,048 and 4,096 keys, at most 148 of
them) and the upward pass's forms (all levels in one launch, eight lanes or one
thread per twig), against a stable sort and the oracle.  Bit equality."""
import numpy as np
import pytest

import pepc_b200 as P
from oracle import oracle as O
from tests.datasets import cube, plummer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tc(gpu):
    t = P.TreeCode()
    yield t
    t.close()


@pytest.mark.parametrize("n", [1, 2, 31, 511, 512, 513, 1023, 1024, 1025, 32768, 32769, 131072, 131073,
                               148 * 4096, 148 * 4096 + 1])
def test_sort_sizes(tc, n):
    # keys over all 64 bits (ordered as unsigned), distinct with all but certainty
    keys = np.random.default_rng(n).integers(-(1 << 63), (1 << 63) - 1, size=n, dtype=np.int64)
    k, p = tc.sort_keys(keys)
    ref = np.argsort(keys.view(np.uint64), kind="stable")
    assert np.array_equal(p, ref)
    assert np.array_equal(k, keys[ref])


@pytest.mark.parametrize("n", [1024, 32769, 131073])
def test_sort_is_stable_in_every_digit(tc, n):
    # few values per digit: long runs of equal digits over every tile boundary
    rng = np.random.default_rng(n)
    keys = np.zeros(n, np.int64)
    for shift in range(0, 60, 3):
        keys |= rng.integers(0, 2, size=n, dtype=np.int64) << shift
    keys = np.unique(keys)
    rng.shuffle(keys)
    k, p = tc.sort_keys(keys)
    assert np.array_equal(p, np.argsort(keys, kind="stable"))
    assert np.array_equal(k, np.sort(keys))


# 1,024 / 131,073 / 606,209: the sort's lines; 230,000 .. 300,000 lie around the widest
# level of 40,000 twigs, 606,209 has levels on both sides of 30,000
@pytest.mark.parametrize("n,data", [(9, "cube"), (1024, "cube"), (1025, "plummer"), (131073, "cube"),
                                    (230011, "plummer"), (300007, "plummer"), (606209, "plummer")])
def test_grow_sizes_match_oracle(gpu, n, data):
    x, y, z, q = cube(n, 61, charges="gauss") if data == "cube" else plummer(n, 62)
    tc, orc = P.TreeCode(), O.Oracle(num_threads=8)
    g, go = tc.pepc_grow_tree(x, y, z, q), orc.grow_tree(x, y, z, q)
    assert np.array_equal(g.key, go["key"])
    assert np.array_equal(g.perm, go["perm"])
    t, to = tc.tree(), orc.tree()
    for k in ("key", "level", "leaves", "descendants", "parent", "first_child", "next_sibling",
              "moments"):
        assert np.array_equal(t[k], to[k]), k
    tc.close()
    orc.close()
