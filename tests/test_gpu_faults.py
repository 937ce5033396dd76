"""GPU: failures made on the host, and the library's recovery from them.

Device allocations fail on demand through pepcg_debug_fail_allocations (a
host-side injection: the allocation call is answered with an error before it
reaches the device).  A grow or traverse that meets the failure must return
PEPCG_ERR_OOM with a message, leave no tree behind, and the same context must
then work again and give the results of a fresh context.

The grid barriers of the cooperative kernels give up at once with no tries
(pepcg_debug_barrier_tries): the call that needed one must return
PEPCG_ERR_TIMEOUT, read nothing that the kernel did not write, and the context
must work again."""
import numpy as np
import pytest

import pepc_b200 as P
from tests.datasets import cube

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_injection(gpu):
    yield
    P.lib().pepcg_debug_fail_allocations(-1)


@pytest.mark.parametrize("after", [0, 1, 5, 12, 20])
def test_grow_allocation_failure_then_recovery(no_injection, after):
    x, y, z, q = cube(30000, 81, charges="normal")
    ref = P.TreeCode(theta2=0.25, eps2=1e-4)
    g_ref = ref.pepc_grow_tree(x, y, z, q)
    r_ref = ref.pepc_traverse_tree(g_ref.x, g_ref.y, g_ref.z, keys=g_ref.key)
    ref.close()
    tc = P.TreeCode(theta2=0.25, eps2=1e-4)
    P.lib().pepcg_debug_fail_allocations(after)
    with pytest.raises(P.PepcgError) as e:
        tc.pepc_grow_tree(x, y, z, q)
    assert e.value.code == P.PEPCG_ERR_OOM
    assert "injected" in str(e.value)
    P.lib().pepcg_debug_fail_allocations(-1)
    # nothing was grown: a traverse is refused, not run on stale data
    with pytest.raises(P.PepcgError) as e2:
        tc.pepc_traverse_tree(x[:10], y[:10], z[:10])
    assert e2.value.code == P.PEPCG_ERR_NO_TREE
    g = tc.pepc_grow_tree(x, y, z, q)
    r = tc.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key)
    assert np.array_equal(g.perm, g_ref.perm)
    for k in ("ex", "ey", "ez", "pot", "work"):
        assert np.array_equal(r[k], r_ref[k]), k
    tc.close()


def test_traverse_allocation_failure_keeps_the_tree(no_injection):
    x, y, z, q = cube(20000, 82, charges="normal")
    tc = P.TreeCode(theta2=0.25, eps2=1e-4)
    g = tc.pepc_grow_tree(x, y, z, q)
    P.lib().pepcg_debug_fail_allocations(0)
    with pytest.raises(P.PepcgError) as e:
        # foreign targets need staging buffers the grow did not allocate
        tc.pepc_traverse_tree(np.linspace(0, 1, 70000), np.full(70000, 0.5), np.full(70000, 0.5))
    assert e.value.code == P.PEPCG_ERR_OOM
    P.lib().pepcg_debug_fail_allocations(-1)
    r = tc.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key)
    assert np.all(np.isfinite(r["pot"])) and np.all(r["work"] > 0)
    tc.close()


def same_results(tc, x, y, z, q):
    """tc grows and walks as a fresh context does."""
    ref = P.TreeCode(theta2=0.25, eps2=1e-4)
    out = []
    for t in (ref, tc):
        g = t.pepc_grow_tree(x, y, z, q)
        r = t.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key)
        out.append([g.perm, g.key] + [r[k] for k in ("ex", "ey", "ez", "pot", "work")])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    ref.close()


# one tile of the sort is 1,024 keys up to 32,768, 2,048 up to 131,072, then 4,096; up to
# 1,024 keys it has no barrier
@pytest.mark.parametrize("used", [False, True])
@pytest.mark.parametrize("n", [1025, 16411, 100003, 600001])
def test_sort_gives_up_then_recovery(gpu, n, used):
    x, y, z, q = cube(n, 83, charges="normal")
    for a in (x, y, z):  # some equal keys
        a[1:100:2] = a[0:99:2]
    tc = P.TreeCode(theta2=0.25, eps2=1e-4)
    if used:  # else every buffer of the context is fresh memory
        tc.pepc_grow_tree(*cube(n + 1000, 84, charges="normal"))
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    with pytest.raises(P.PepcgError) as e:
        tc.pepc_grow_tree(x, y, z, q)
    assert e.value.code == P.PEPCG_ERR_TIMEOUT
    with pytest.raises(P.PepcgError) as e:
        tc.pepc_traverse_tree(x[:10], y[:10], z[:10])
    assert e.value.code == P.PEPCG_ERR_NO_TREE
    P.lib().pepcg_debug_barrier_tries(tc._h, -1)
    same_results(tc, x, y, z, q)
    tc.close()


@pytest.mark.parametrize("n", [1025, 30011])
def test_key_sort_gives_up_then_recovery(gpu, n):
    keys = np.random.default_rng(85).integers(0, n // 2, n)  # with equal keys
    tc = P.TreeCode()
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    with pytest.raises(P.PepcgError) as e:
        tc.sort_keys(keys)
    assert e.value.code == P.PEPCG_ERR_TIMEOUT
    P.lib().pepcg_debug_barrier_tries(tc._h, -1)
    ko, po = tc.sort_keys(keys)
    assert np.array_equal(ko, np.sort(keys)) and np.array_equal(keys[po], ko)
    tc.close()


WALKS = [(P.PRECISION_PLAIN, P.WALK_PER_TARGET), (P.PRECISION_PLAIN, P.WALK_PER_TILE),
         (P.PRECISION_PLAIN, P.WALK_GROUP), (P.PRECISION_MIXED, P.WALK_PER_TARGET),
         (P.PRECISION_MIXED, P.WALK_PER_TILE), (P.PRECISION_MIXED, P.WALK_GROUP),
         (P.PRECISION_MIXED_STRICT, P.WALK_GROUP)]


@pytest.mark.parametrize("precision,walk", WALKS)
def test_upward_pass_gives_up_and_every_reader_says_so(gpu, precision, walk):
    # up to 1,024 keys the sort has no barrier and the scans (one tile) have none, the
    # upward pass has: the grow returns before it
    x, y, z, q = cube(1000, 86, charges="normal")
    kw = dict(theta2=0.25, eps2=1e-4, precision=precision, walk=walk)
    tc, ref = P.TreeCode(**kw), P.TreeCode(**kw)
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    g = tc.pepc_grow_tree(x, y, z, q)
    zero, one = np.zeros(1000), np.ones(1000)
    for call in (lambda: tc.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key),
                 lambda: tc.traverse_adjoint(g.x, g.y, g.z, [zero] * 3, one, 1000),
                 tc.tree):
        with pytest.raises(P.PepcgError) as e:
            call()
        assert e.value.code == P.PEPCG_ERR_TIMEOUT
    P.lib().pepcg_debug_barrier_tries(tc._h, -1)
    tc.pepc_grow_tree(x, y, z, q)
    ref.pepc_grow_tree(x, y, z, q)
    a, b = [t.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key) for t in (tc, ref)]
    assert all(np.array_equal(a[k], b[k]) for k in ("ex", "ey", "ez", "pot", "work"))
    tc.close()
    ref.close()


def test_group_walk_by_warps_leaves_an_unbuilt_tree_alone(gpu):
    # more buckets than the walk by blocks takes
    n, nt = 1000, 9000 * 64 + 1
    tc = P.TreeCode(theta2=0.25, eps2=1e-4, precision=P.PRECISION_MIXED, walk=P.WALK_GROUP)
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    tc.pepc_grow_tree(*cube(n, 87, charges="normal"))
    t = np.random.default_rng(88).random((3, nt))
    with pytest.raises(P.PepcgError) as e:
        tc.pepc_traverse_tree(*t)
    assert e.value.code == P.PEPCG_ERR_TIMEOUT
    tc.close()


@pytest.mark.parametrize("precision,walk", WALKS)
def test_downward_pass_gives_up_in_the_host_adjoint(gpu, precision, walk):
    n = 3000
    x, y, z, q = cube(n, 89, charges="normal")
    tc = P.TreeCode(theta2=0.25, eps2=1e-4, precision=precision, walk=walk)
    g = tc.pepc_grow_tree(x, y, z, q)
    args = (g.x, g.y, g.z, [np.zeros(n)] * 3, np.ones(n), n)
    good = tc.traverse_adjoint(*args)
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    with pytest.raises(P.PepcgError) as e:
        tc.traverse_adjoint(*args)
    assert e.value.code == P.PEPCG_ERR_TIMEOUT and "adjoint" in str(e.value)
    P.lib().pepcg_debug_barrier_tries(tc._h, -1)
    again = tc.traverse_adjoint(*args)
    # FP64 atomics: each sum's some 1e4 terms in another order, 1e4 * 2^-53 of terms that
    # may cancel to a thousandth
    for k in good:
        assert np.abs(again[k] - good[k]).max() <= 1e-9 * np.abs(good[k]).max(), k
    tc.close()


@pytest.mark.parametrize("after", ["grow", "traverse", "adjoint", "export"])
def test_next_call_reports_a_device_adjoint_that_gave_up(gpu, after):
    import torch
    n = 3000
    p = [torch.from_numpy(v).cuda() for v in cube(n, 90, charges="normal")]
    tc = P.TreeCode(theta2=0.25, eps2=1e-4, precision=P.PRECISION_MIXED, walk=P.WALK_GROUP)
    tc.set_stream(torch.cuda.current_stream().cuda_stream)
    tc.grow_tree_device(*p)
    f = torch.zeros((9, n), dtype=torch.float64, device="cuda")
    calls = dict(grow=lambda: tc.grow_tree_device(*p),
                 traverse=lambda: tc.traverse_self_device(*f[:5]),
                 adjoint=lambda: tc.traverse_adjoint_device(*p[:3], [f[5]] * 3, torch.ones_like(f[5]),
                                                            *f[:4]),
                 export=tc.tree)
    P.lib().pepcg_debug_barrier_tries(tc._h, 0)
    calls["adjoint"]()  # returns while its kernels run
    P.lib().pepcg_debug_barrier_tries(tc._h, -1)
    with pytest.raises(P.PepcgError) as e:
        calls[after]()
    assert e.value.code == P.PEPCG_ERR_TIMEOUT and "adjoint" in str(e.value)
    for k in ("grow", "traverse", "adjoint", "export", "grow"):  # reported once
        calls[k]()
    tc.close()


@pytest.mark.parametrize("precision", [P.PRECISION_PLAIN, P.PRECISION_MIXED])
def test_refused_walk_stream_then_recovery(gpu, precision):
    n = 300001  # host targets in chunks, on two streams
    x, y, z, q = cube(n, 91, charges="normal")
    kw = dict(theta2=0.36, eps2=1e-4, precision=precision, walk=P.WALK_GROUP)
    tc, ref = P.TreeCode(**kw), P.TreeCode(**kw)
    P.lib().pepcg_debug_refuse(tc._h, 1)
    for _ in range(2):
        with pytest.raises(P.PepcgError) as e:
            tc.pepc_grow_tree(x, y, z, q)
        assert e.value.code == P.PEPCG_ERR_CUDA and "walk stream" in str(e.value)
    P.lib().pepcg_debug_refuse(tc._h, 0)
    out = []
    for t in (tc, ref):
        g = t.pepc_grow_tree(x, y, z, q)
        out.append(t.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key))
    assert all(np.array_equal(out[0][k], out[1][k]) for k in ("ex", "ey", "ez", "pot", "work"))
    tc.close()
    ref.close()


def tree_bits(t):
    return {k: (v.view(np.int64) if v.dtype == np.float64 else v) for k, v in t.tree().items()}


# sizes: each tile width of the one-launch sort and both forms of the upward pass
@pytest.mark.parametrize("n", [1000, 16411, 100003, 600001])
def test_refused_cooperative_launches_give_the_same_tree(gpu, n):
    x, y, z, q = cube(n, 92, charges="normal")
    tc, ref = P.TreeCode(theta2=0.36, eps2=1e-4), P.TreeCode(theta2=0.36, eps2=1e-4)
    P.lib().pepcg_debug_refuse(tc._h, 2)
    launches, got = [], []
    for t in (ref, tc):
        a = P.lib().pepcg_kernel_launches()
        g = t.pepc_grow_tree(x, y, z, q)
        launches.append(P.lib().pepcg_kernel_launches() - a)
        got.append((g.key, g.perm, tree_bits(t), t.sort_keys(g.key[::-1]),
                    t.traverse_adjoint(x[:300], y[:300], z[:300], [np.zeros(300)] * 3, np.ones(300), n)))
    assert launches[1] > launches[0]
    a, b = got
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert all(np.array_equal(a[2][k], b[2][k]) for k in a[2])
    assert all(np.array_equal(u, v) for u, v in zip(a[3], b[3]))
    for k in a[4]:  # FP64 atomics, as above
        assert np.abs(a[4][k] - b[4][k]).max() <= 1e-9 * np.abs(a[4][k]).max(), k
    tc.close()
    ref.close()


# clusters of eight blocks of sixteen and of eight warps, of four blocks
@pytest.mark.parametrize("n,nt", [(40000, 1000), (5000, 1000), (5000, 2000), (5000, 4000)])
@pytest.mark.parametrize("precision", [P.PRECISION_MIXED, P.PRECISION_MIXED_STRICT])
def test_refused_cluster_launches_walk_by_warps(gpu, precision, n, nt):
    x, y, z, q = cube(n, 93, charges="normal")
    t = np.random.default_rng(94).random((3, nt))
    kw = dict(theta2=0.25, eps2=1e-4, precision=precision, walk=P.WALK_GROUP)
    got = []
    for refuse in (0, 4):
        tc = P.TreeCode(**kw)
        P.lib().pepcg_debug_refuse(tc._h, refuse)
        tc.pepc_grow_tree(x, y, z, q)
        got.append((tc.pepc_traverse_tree(*t),
                    tc.traverse_adjoint(*t, [np.zeros(nt)] * 3, np.ones(nt), n)))
        tc.close()
    # the same lists (one opening test); the sums differ in order: FP32 within batches of
    # 32, a few 2^-24 of terms that may cancel to a hundredth
    (f, a), (g, b) = got
    assert np.array_equal(f["work"], g["work"])
    for u, v, keys in ((f, g, ("ex", "ey", "ez", "pot")), (a, b, ("q", "x", "y", "z"))):
        for k in keys:
            assert np.abs(u[k] - v[k]).max() <= 1e-5 * np.abs(u[k]).max(), k
