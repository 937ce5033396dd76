"""GPU: the adjoint's downward pass at tree sizes around its forms (all levels in one
launch with one block, with many, level by level), by an identity: with the lists and the
abs_charge-weighted centres fixed under a common factor of the charges, the loss is
homogeneous of degree one in them, so sum q dL/dq = L.  FP64 walks: 1e-10 of the
sum of |q dL/dq| (some hundred thousand terms, atomic order)."""
import numpy as np
import pytest
import torch

import pepc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 9, 130, 3001, 40009, 250007, 1300001])
def test_charges_scale_the_loss(gpu, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    f = dict(dtype=torch.float64, device="cuda")
    p = torch.rand((3, n), generator=g, **f)
    q = torch.randn(n, generator=g, **f)
    t = torch.rand((3, 300), generator=g, **f)
    gr = torch.randn((4, 300), generator=g, **f)
    tc = P.TreeCode(theta2=0.25, eps2=1e-4)
    tc.set_stream(torch.cuda.current_stream().cuda_stream)
    tc.grow_tree_device(*p, q)
    out = torch.zeros((5, 300), **f)
    tc.traverse_tree_device(*t, *out)
    loss = (gr * out[:4]).sum()
    o = torch.empty((4, n), **f)
    tc.traverse_adjoint_device(*t, [gr[0], gr[1], gr[2]], gr[3], *o)
    terms = q * o[0]
    assert float((terms.sum() - loss).abs()) <= 1e-10 * float(terms.abs().sum())
    # a common shift of the sources moves the fields as the opposite shift of the targets:
    # sum dL/dx against a central difference of the loss over the targets' positions,
    # at a step below which no list changes but for one in 1e5 nodes: a target whose list
    # does (its length tells) has no part in the loss
    h = 1e-6
    for d in range(3):
        s = []
        for sign in (1, -1):
            tt = t.clone()
            tt[d] += sign * h
            w = torch.zeros((5, 300), **f)
            tc.traverse_tree_device(*tt, *w)
            s.append(w)
        same = (s[0][4] == out[4]) & (s[1][4] == out[4])
        assert int(same.sum()) >= 290, (n, d)
        gs = gr * same
        fd = ((gs * s[0][:4]).sum() - (gs * s[1][:4]).sum()) / (2 * h)
        tc.traverse_adjoint_device(*t, [gs[0], gs[1], gs[2]], gs[3], *o)
        scale = o[1 + d].abs().sum()
        assert float((o[1 + d].sum() + fd).abs()) <= 1e-6 * float(scale)
    tc.close()


MODES = [(P.PRECISION_PLAIN, P.WALK_PER_TARGET), (P.PRECISION_PLAIN, P.WALK_PER_TILE),
         (P.PRECISION_PLAIN, P.WALK_GROUP), (P.PRECISION_MIXED, P.WALK_PER_TARGET),
         (P.PRECISION_MIXED, P.WALK_GROUP), (P.PRECISION_MIXED_STRICT, P.WALK_GROUP)]


@pytest.mark.parametrize("precision,walk", MODES)
def test_no_targets_give_zero_gradients(gpu, precision, walk):
    rng = np.random.default_rng(3)
    none = np.zeros(0)
    tc = P.TreeCode(theta2=0.25, eps2=1e-4, precision=precision, walk=walk)
    tc.pepc_grow_tree(*rng.random((3, 500)), rng.standard_normal(500))
    r = tc.traverse_adjoint(none, none, none, [none] * 3, none, 500)
    assert all(np.array_equal(r[k], np.zeros(500)) for k in ("q", "x", "y", "z"))
    tc.close()
