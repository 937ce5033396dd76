"""GPU: the 64-target group walk and its adjoint by one block or cluster per
bucket (walk_block.cu), at the target counts where the choice of the block's
warps and blocks changes and at ragged last buckets, against the FP64 group walk
with the same buckets.

Tolerances: the strict form takes the FP64 walk's decisions, so work is equal;
a field is a sum of some thousand FP32 terms of relative error a few 2^-24, added
in FP64 per batch of 32, hence 2e-6 (median) and 1e-5 of the fields' scale; the
default form's offsets add the term derived at its check."""
import numpy as np
import pytest
import torch

import pepc_b200 as P

pytestmark = pytest.mark.gpu

EDGES = [1, 63, 64, 65, 18 * 64, 18 * 64 + 1, 37 * 64, 37 * 64 + 1, 74 * 64, 74 * 64 + 1, 148 * 64,
         148 * 64 + 1, 600 * 64 + 1, 5000 * 64 + 1, 9000 * 64 + 1]


def sources(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    p = torch.rand((3, n), generator=g, dtype=torch.float64, device="cuda")
    return [*p, torch.randn(n, generator=g, dtype=torch.float64, device="cuda")], g


def targets(nt, g):
    t = torch.rand((3, nt), generator=g, dtype=torch.float64, device="cuda")
    return [r.contiguous() for r in t[:, torch.argsort(t[0])]]  # buckets are slabs


def context(p, **kw):
    tc = P.TreeCode(walk=P.WALK_GROUP, group_size=64, **kw)
    tc.set_stream(torch.cuda.current_stream().cuda_stream)
    tc.grow_tree_device(*p)
    return tc


def fields(tc, t):
    out = torch.zeros((5, t[0].numel()), dtype=torch.float64, device="cuda")
    tc.traverse_tree_device(*t, *out)
    return out


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("n", [2500, 33000])
def test_block_walk_matches_fp64_lists(gpu, n, periodic):
    p, g = sources(n, 11)
    kw = dict(theta2=0.25, eps2=1e-6)
    if periodic:  # 27 boxes, no far field: the walk alone
        kw.update(periodicity=(1, 1, 1), include_far_field_if_periodic=0)
    plain = context(p, precision=P.PRECISION_PLAIN, **kw)
    for prec in (P.PRECISION_MIXED, P.PRECISION_MIXED_STRICT):
        tc = context(p, precision=prec, **kw)
        for nt in EDGES:
            if nt > 40000 and (periodic or n > 10000):
                continue  # 38,401 targets, the first count of four-warp blocks, are in
            t = targets(nt, g)
            a, b = fields(plain, t), fields(tc, t)
            if prec == P.PRECISION_MIXED_STRICT:
                assert torch.equal(a[4], b[4]), nt
            scale = a[:3].norm(dim=0).median()
            off = (a[:3] - b[:3]).norm(dim=0) / torch.maximum(a[:3].norm(dim=0), scale)
            assert float(off.median()) < 2e-6, (nt, float(off.median()))
            same = a[4] == b[4]  # the default form may decide a node on the threshold otherwise
            assert float(same.double().mean()) > 0.98, nt
            # largest: the default form's offsets carry 2^-23 r_g (r_g <= 0.9, a slab of
            # the cube) against a nearest source at ~1e-3 (eps and 5e8 pairs): 3 of them
            # (E goes with |d|^-3) are 3.2e-4.  The strict form rounds FP64 offsets
            worst = 1e-5 if prec == P.PRECISION_MIXED_STRICT else 5e-4
            assert float(off[same].max()) < worst, (nt, float(off[same].max()))
            again = fields(tc, t)
            assert torch.equal(again, b), nt  # a fixed order of summation
        tc.close()
    plain.close()


@pytest.mark.parametrize("precision,lines", [(P.PRECISION_MIXED, (4096, 9000)),
                                             (P.PRECISION_MIXED_STRICT, (2200, 2368, 5000))])
def test_targets_with_and_without_keys(gpu, precision, lines):
    # without keys other bucket counts go by blocks: the same lists, and sums that differ in
    # order (FP32 in batches of 32, then FP64: a few 2^-24 of terms that cancel to a tenth)
    p, _ = sources(2500, 15)
    tc = context(p, precision=precision, theta2=0.25, eps2=1e-4)
    q = [torch.empty(2500, dtype=torch.float64, device="cuda") for _ in range(4)]
    k = torch.empty((2, 2500), dtype=torch.int64, device="cuda")
    tc.particles_device(*k, *q)
    for nb in lines:
        for nt in (64 * nb - 63, 64 * nb + 1):
            i = torch.arange(nt, device="cuda") * 2500 // nt  # in key order
            t, keys = [a[i].contiguous() for a in q[:3]], k[0][i].contiguous()
            a = fields(tc, t)
            b = torch.zeros_like(a)
            tc.traverse_tree_device(*t, *b, keys=keys)
            assert torch.equal(a[4], b[4]), nt
            scale = a[:3].norm(dim=0).median()
            off = (a[:3] - b[:3]).norm(dim=0) / torch.maximum(a[:3].norm(dim=0), scale)
            assert float(off.max()) < 5e-6, (nt, float(off.max()))
    tc.close()


@pytest.mark.parametrize("with_e", [False, True])
@pytest.mark.parametrize("n", [2500, 33000])
def test_block_adjoint_matches_fp64(gpu, n, with_e):
    p, g = sources(n, 12)
    kw = dict(theta2=0.25, eps2=1e-4)
    plain = context(p, precision=P.PRECISION_PLAIN, **kw)
    tc = context(p, precision=P.PRECISION_MIXED, **kw)
    for nt in EDGES + [6000 * 64 + 1]:
        if nt > 40000 and n > 10000:
            continue
        t = targets(nt, g)
        gr = torch.randn((4, nt), generator=g, dtype=torch.float64, device="cuda")
        if not with_e:
            gr[:3] = 0.0
        res = []
        for c in (plain, tc):
            o = torch.empty((4, n), dtype=torch.float64, device="cuda")
            c.traverse_adjoint_device(*t, [gr[0], gr[1], gr[2]], gr[3], *o)
            res.append(o)
        a, b = res
        for k in range(4):
            off = (a[k] - b[k]).abs() / a[k].abs().max()
            assert float(off.median()) < 1e-6, (nt, k, float(off.median()))
            assert float((a[k] - b[k]).norm() / a[k].norm()) < 1e-4, (nt, k)
    plain.close()
    tc.close()


@pytest.mark.parametrize("n", [4099, 30011, 100003])
def test_ranges_equal_the_single_call(gpu, n):
    # a share of the targets takes the kernel of the whole set: equal bits
    p, _ = sources(n, 13)
    for prec in (P.PRECISION_MIXED, P.PRECISION_MIXED_STRICT):
        tc = context(p, precision=prec, theta2=0.25, eps2=1e-6)
        whole = torch.zeros((5, n), dtype=torch.float64, device="cuda")
        tc.traverse_self_device(*whole)
        t0 = 0
        for t1 in (64, n // 3 // 64 * 64, n):
            part = torch.zeros((5, t1 - t0), dtype=torch.float64, device="cuda")
            tc.traverse_range_device(t0, t1, *part)
            assert torch.equal(part, whole[:, t0:t1]), (t0, t1)
            t0 = t1
        tc.close()


def test_bucket_results_accumulate(gpu):
    p, g = sources(2500, 14)
    tc = context(p, precision=P.PRECISION_MIXED, theta2=0.25, eps2=1e-6)
    t = targets(700, g)
    once = fields(tc, t)
    twice = once.clone()
    tc.traverse_tree_device(*t, *twice)
    assert torch.equal(twice[4], 2 * once[4])
    assert float((twice - 2 * once).abs().max()) <= 1e-12 * float(once.abs().max())
    tc.close()


def test_more_nodes_than_a_packed_stack_entry_holds(gpu):
    # above 2^25 nodes the image boxes are swept one after the other: the fields of 27 boxes
    # against 27 walks of the open tree by shifted targets (the same lists but where the
    # shift's rounding decides a node otherwise)
    n = 24_000_000
    p, g = sources(n, 16)
    kw = dict(precision=P.PRECISION_MIXED, theta2=0.25, eps2=1e-6)
    targets_of = [targets(nt, g) for nt in (500, 9000)]  # clusters, and one block per bucket
    tc = context(p, periodicity=(1, 1, 1), include_far_field_if_periodic=0, **kw)
    assert P.lib().pepcg_num_nodes(tc._h) > 2 ** 25
    boxes = [fields(tc, t) for t in targets_of]
    tc.close()
    tc = context(p, **kw)
    for t, a in zip(targets_of, boxes):
        b = torch.zeros_like(a)
        for i in range(27):
            tc.traverse_tree_device(*[c + (i // 3 ** k % 3 - 1) for k, c in enumerate(t)], *b)
        assert float(((a[4] - b[4]).abs() / b[4]).max()) < 1e-3
        off = (a[:3] - b[:3]).norm(dim=0) / b[:3].norm(dim=0).median()
        assert float(off.median()) < 2e-6, float(off.median())
        assert float(off.max()) < 5e-4, float(off.max())
    tc.close()
