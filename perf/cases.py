"""The work that is timed: force evaluations, gradients and host calls of the
tree code, from a thousand particles to the 4M-particle configuration, each
through the calls a program makes (pepc_b200.TreeCode).

A case's "kind":
  step  one step of a device-resident simulation: results cleared, the tree
        grown from the particles, the fields of all particles (both the mixed
        group walk and the FP64 walks, open and periodic boundaries);
  fit   one step of fitting source charges and positions to potentials measured
        at probe points: grow, potentials at the probes, the adjoint of the
        squared loss (dL/dq, dL/dx of the sources);
  grad  the adjoint for the particles' own fields: grow, fields, and the
        gradient of a loss with given dL/dE and dL/dphi at every particle;
  host  the drop-in calls on host arrays (grow, then traverse), as a CPU
        frontend makes them.

exact() evaluates the same tree code in plain torch, in 64 bits: octree cells
from sorted keys, moments as sums over each cell's particles, and every
target's (or target group's) interaction list by the opening criterion.
"""
import functools
import math

import numpy as np
import torch

import pepc_b200

MAXLEVEL = 20
NO_EXACT_ABOVE = 400_000  # particles: the 64-bit evaluation would take too long

# precision, walk, targets that share one list (0: tiles of at most 16)
MODES = {
    "mixed": (pepc_b200.PRECISION_MIXED, pepc_b200.WALK_GROUP, 64),
    "strict": (pepc_b200.PRECISION_MIXED_STRICT, pepc_b200.WALK_GROUP, 64),
    "plain": (pepc_b200.PRECISION_PLAIN, pepc_b200.WALK_PER_TARGET, 1),
    "tile": (pepc_b200.PRECISION_PLAIN, pepc_b200.WALK_PER_TILE, 0),
}


def listed():
    return [
        # a small system stepped many thousand times: launches and latency count
        dict(name="step_mixed_1k", kind="step", mode="mixed", n=1000, dist="plummer", theta=0.4),
        # a laboratory-sized run, an odd particle count
        dict(name="step_mixed_16k", kind="step", mode="mixed", n=16411, dist="cube", theta=0.6),
        # an ordinary production step
        dict(name="step_mixed_200k", kind="step", mode="mixed", n=200003, dist="plummer", theta=0.4),
        # the clustered-gravity configuration of bench.py
        dict(name="step_mixed_4m", kind="step", mode="mixed", n=4194304, dist="plummer", theta=0.4),
        # the precision form with FP64 offsets and compensated sums
        dict(name="step_strict_60k", kind="step", mode="strict", n=60013, dist="plummer", theta=0.4),
        # the FP64 drop-in, default parameters: a small and a medium run
        dict(name="step_plain_4k", kind="step", mode="plain", n=4099, dist="cube", theta=0.6),
        dict(name="step_plain_250k", kind="step", mode="plain", n=250000, dist="plummer", theta=0.6),
        # the other reference walk (shared lists for tiles of 16)
        dict(name="step_tile_40k", kind="step", mode="tile", n=40009, dist="cube", theta=0.6),
        # ions near a rock-salt lattice, periodic in all directions with the far-lattice term
        dict(name="step_periodic_33k", kind="step", mode="mixed", n=32768, dist="ions", theta=0.3),
        # the adjoint configuration: 262,144 sources, 4,096 probes, potentials only
        dict(name="fit_262k_4k", kind="fit", mode="mixed", n=262144, nt=4096, theta=0.4),
        # gradient of a loss on every particle's field and potential
        dict(name="grad_100k", kind="grad", mode="mixed", n=100003, dist="plummer", theta=0.4),
        # a CPU frontend's step on host arrays, default parameters
        dict(name="host_plain_30k", kind="host", mode="plain", n=30011, dist="cube", theta=0.6),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["mixed", "mixed", "mixed", "strict", "plain", "plain", "tile", "ions", "fit",
                       "grad", "host"])
    theta = round(rng.uniform(0.35, 0.65), 2)
    dist = rng.choice(["plummer", "cube"])
    if kind == "ions":
        return dict(kind="step", mode="mixed", n=(2 * rng.randint(5, 22)) ** 3, dist="ions",
                    theta=round(rng.uniform(0.3, 0.6), 2))
    if kind == "fit":
        return dict(kind="fit", mode="mixed", n=size(8000, 400000), nt=size(500, 8000), theta=theta)
    if kind == "grad":
        return dict(kind="grad", mode="mixed", n=size(2000, 300000), dist=dist, theta=theta)
    if kind == "host":
        return dict(kind="host", mode=rng.choice(["plain", "mixed"]), n=size(1000, 200000), dist=dist,
                    theta=theta)
    hi = {"mixed": 2000000, "strict": 500000, "plain": 500000, "tile": 300000}[kind]
    return dict(kind="step", mode=kind, n=size(1000, hi), dist=dist, theta=theta)


# ---- inputs ----
def _gen(seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _eps2(case):
    return 0.0 if case.get("dist") == "ions" else 1.0e-6


def _particles(case, seed):
    """x, y, z, q as FP64 tensors on the GPU."""
    dev = torch.device("cuda")
    n, g = case["n"], _gen(seed, dev)
    f = dict(dtype=torch.float64, device=dev)
    if case["kind"] == "fit":  # sources uniform in the unit cube, charges N(0, 1)
        p = torch.rand((3, n), generator=g, **f)
        q = torch.randn(n, generator=g, **f)
    elif case["dist"] == "plummer":  # a = 1, r <= 20, equal masses
        u = torch.rand(n, generator=g, **f) * (20.0 ** 3 / (1.0 + 400.0) ** 1.5)
        u = u.clamp_min(1e-12)
        r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
        v = torch.randn((3, n), generator=g, **f)
        p = v * (r / v.norm(dim=0))
        q = torch.full((n,), 1.0 / n, **f)
    elif case["dist"] == "ions":  # rock salt in the unit cube, thermal displacements
        m = round(n ** (1.0 / 3.0))
        i = torch.arange(m, device=dev)
        i, j, k = torch.meshgrid(i, i, i, indexing="ij")
        p = (torch.stack([i, j, k]).reshape(3, -1).to(torch.float64) + 0.5) / m
        p = (p + torch.randn((3, n), generator=g, **f) * (0.08 / m)).clamp(1e-9, 1.0 - 1e-9)
        q = 1.0 - 2.0 * ((i + j + k).reshape(-1) % 2).to(torch.float64)
    else:  # uniform in the unit cube, alternating charges
        p = torch.rand((3, n), generator=g, **f)
        q = 1.0 - 2.0 * (torch.arange(n, device=dev) % 2).to(torch.float64)
    return p[0].contiguous(), p[1].contiguous(), p[2].contiguous(), q


def _loss(case, seed):
    """fit: probe positions (3, nt) and measured potentials; grad: dL/dE (3, n), dL/dphi."""
    dev = torch.device("cuda")
    g = _gen(seed + 1000003, dev)
    f = dict(dtype=torch.float64, device=dev)
    if case["kind"] == "fit":
        t = 0.25 + 0.5 * torch.rand((3, case["nt"]), generator=g, **f)
        return t, torch.randn(case["nt"], generator=g, **f) * math.sqrt(case["n"])
    return (torch.randn((3, case["n"]), generator=g, **f),
            torch.randn(case["n"], generator=g, **f))


def prepare(case, seed):
    precision, walk, _ = MODES[case["mode"]]
    kw = dict(theta2=case["theta"] ** 2, eps2=_eps2(case), precision=precision, walk=walk)
    if case.get("dist") == "ions":
        kw.update(periodicity=(1, 1, 1))
    if case["kind"] == "host":
        kw.update(overwrite_results=1)  # the frontend clears its results before each step
    tc = pepc_b200.TreeCode(**kw)
    p = _particles(case, seed)
    s = dict(case=case, tc=tc)
    if case["kind"] == "host":
        s["p"] = [a.cpu().numpy() for a in p]
        return s
    tc.set_stream(torch.cuda.current_stream().cuda_stream)
    s["p"] = p
    nt = case["nt"] if case["kind"] == "fit" else case["n"]
    s["out"] = torch.zeros((5, nt), dtype=torch.float64, device="cuda")  # ex ey ez pot work
    if case["kind"] in ("fit", "grad"):
        a, b = _loss(case, seed)
        s["grad"] = torch.empty((4, case["n"]), dtype=torch.float64, device="cuda")
        s["a"], s["b"] = [r.contiguous() for r in a], b
        s["zero"] = torch.zeros(nt, dtype=torch.float64, device="cuda")
        s["xk"] = torch.empty((4, case["n"]), dtype=torch.float64, device="cuda")
        s["key"] = torch.empty((2, case["n"]), dtype=torch.int64, device="cuda")
    return s


def run(s):
    case, tc, p = s["case"], s["tc"], s["p"]
    if case["kind"] == "host":
        g = tc.pepc_grow_tree(*p)
        r = tc.pepc_traverse_tree(g.x, g.y, g.z, keys=g.key)
        return dict(r, key=g.key, perm=g.perm)
    out = s["out"]
    out.zero_()
    tc.grow_tree_device(*p)
    if case["kind"] == "step":
        tc.traverse_self_device(*out)
        return dict(e=out[:3], pot=out[3], work=out[4])
    if case["kind"] == "fit":
        t = s["a"]
        tc.traverse_tree_device(*t, *out)
        dphi = 2.0 * (out[3] - s["b"])
        z = s["zero"]
        tc.traverse_adjoint_device(*t, (z, z, z), dphi, *s["grad"])
        return dict(pot=out[3], work=out[4], dq=s["grad"][0], dx=s["grad"][1:])
    tc.traverse_self_device(*out)
    tc.particles_device(*s["key"], *s["xk"])
    tc.traverse_adjoint_device(*s["xk"][:3], s["a"], s["b"], *s["grad"])
    return dict(e=out[:3], pot=out[3], dq=s["grad"][0], dx=s["grad"][1:])


# ---- what a pass cannot do without ----
def _interactions(n, theta):
    """Interactions per target of a Barnes-Hut walk with its own list: a count per
    octave of distance that goes with theta^-3 (3.9 k at 4M and theta 0.4)."""
    return min(float(n), 23.0 / theta ** 3 * math.log(1.0 + n * theta ** 3 / 4.6))


def work(case):
    n, theta = case["n"], case["theta"]
    nt = case["nt"] if case["kind"] == "fit" else n
    per = _interactions(n, theta)
    flops = nt * per * 75.0 + n * 400.0  # quadrupole interaction; keys, sort, moments
    by = n * 32.0 + nt * 40.0
    if case.get("dist") == "ions":
        # image boxes: most are accepted whole or in a few cells; the near ones add to the list
        flops = nt * per * 2.0 * 75.0 + nt * 231 * 14.0 + n * 231 * 8.0
    if case["kind"] == "fit":
        flops += nt * per * 110.0
        by += nt * 40.0 + n * 32.0
    if case["kind"] == "grad":
        flops += nt * per * 180.0
        by += nt * 32.0 + n * 32.0
    if case["kind"] == "host":
        by += n * 16.0
    return {"bytes": by, "flops": flops}


def tolerance(case):
    """What sums in another order give.  The FP64 walks fix the order of each
    target's sum, so they agree to FP64 rounding; mixed: FP32 interactions, and
    a group whose opening test lands within FP32 rounding of the threshold."""
    if case["mode"] in ("plain", "tile"):
        return {"rel": 1e-12, "max": 1e-9}
    if case.get("dist") == "ions":
        return {"rel": 8e-6, "max": 1e-3}
    if case["kind"] in ("fit", "grad"):
        return {"rel": 8e-6, "max": 1e-3}
    return {"rel": 4e-6, "max": 1e-3}


# ---- the 64-bit evaluation ----
_CI3 = (0, 1, 3, 2, 7, 6, 4, 5)  # octant -> curve digit, and the axes exchanged / reversed below it
_EXCHANGE = (5, 6, 0, 5, 5, 0, 6, 5)
_REVERSE = (0, 0, 0, 5, 0, 0, 6, 5)


def _keys(p):
    """The 60 bits of the Hilbert key of every particle, and the box edges."""
    lo, hi = p.amin(1), p.amax(1)
    lo, hi = lo - (hi - lo) / 10000.0, hi + (hi - lo) / 10000.0
    size = hi - lo
    ic = ((p - lo[:, None]) / (size / 2.0 ** MAXLEVEL)[:, None]).to(torch.int64)
    c = [ic[0], ic[1], ic[2]]
    ci, ex, rv = (torch.tensor(v, device=p.device) for v in (_CI3, _EXCHANGE, _REVERSE))
    key = torch.zeros_like(c[0])
    for i in range(MAXLEVEL - 1, -1, -1):
        h = ci[((c[2] >> i) & 1) << 2 | ((c[1] >> i) & 1) << 1 | (c[0] >> i) & 1]
        key = key << 3 | h
        e, r = ex[h], rv[h]
        a, b = e == 5, e == 6
        c = [torch.where(a, c[2], c[0]), torch.where(b, c[2], c[1]),
             torch.where(a, c[0], torch.where(b, c[1], c[2]))]
        c = [torch.where((r >> j & 1) == 1, ~c[j], c[j]) for j in range(3)]
    return key, size


class _Tree:
    """Octree cells of the key-ordered particles: level by level in key order,
    a cell below every cell of two or more particles."""

    def __init__(self, p, q):
        dev = p.device
        key, size = _keys(p.detach())
        key, self.perm = torch.sort(key, stable=True)
        self.p, self.q = p[:, self.perm], q[self.perm]
        n = key.numel()
        self.n = n
        bl = size.max() ** 2
        part = torch.arange(n, device=dev)       # particles whose cell of this level exists
        start, count, level, first, nch = [], [], [], [], []
        members = []                              # (particle, cell) pairs of every level
        total = 0
        parent_of = None
        for lv in range(MAXLEVEL + 1):
            pre = key[part] >> (3 * (MAXLEVEL - lv))
            _, inv, cnt = torch.unique_consecutive(pre, return_inverse=True, return_counts=True)
            m = cnt.numel()
            st = part[torch.cumsum(cnt, 0) - cnt]
            if parent_of is not None:             # children of the level above: runs in key order
                par = parent_of[st]
                f = torch.searchsorted(par, self._open, right=False) + total
                k = torch.searchsorted(par, self._open, right=True) + total - f
                first[-1][self._open_at], nch[-1][self._open_at] = f, k
            start.append(st)
            count.append(cnt)
            level.append(torch.full((m,), lv, device=dev))
            first.append(torch.zeros(m, dtype=torch.int64, device=dev))
            nch.append(torch.zeros(m, dtype=torch.int64, device=dev))
            members.append((part, inv + total))
            many = cnt > 1
            self._open_at = torch.nonzero(many).flatten()
            self._open = self._open_at + total
            keep = many[inv]
            parent_of = torch.zeros(n, dtype=torch.int64, device=dev)
            parent_of[part] = inv + total
            part = part[keep]
            total += m
            if part.numel() == 0:
                break
        else:
            raise RuntimeError("equal keys")
        self.start, self.count, self.level = (torch.cat(v) for v in (start, count, level))
        self.first, self.nch = torch.cat(first), torch.cat(nch)
        self.bl2 = bl / 4.0 ** self.level.to(torch.float64)
        self.cells = total
        zero = torch.zeros(total, dtype=p.dtype, device=dev)
        a = self.q.abs()

        def sums(value):
            s = zero
            for i, c in members:
                s = s.index_add(0, c, value(i, c))
            return s

        w = sums(lambda i, c: a[i])
        self.coc = torch.stack([sums(lambda i, c: a[i] * self.p[d][i]) / w for d in range(3)])
        leaf = self.count == 1
        at = self.start[leaf]
        self.coc = self.coc.index_copy(1, torch.nonzero(leaf).flatten(), self.p[:, at])
        self.charge = sums(lambda i, c: self.q[i])

        def off(d, i, c):
            return self.coc[d][c] - self.p[d][i]

        self.dip = torch.stack([sums(lambda i, c: self.q[i] * off(d, i, c)) for d in range(3)])
        self.quad = torch.stack(
            [sums(lambda i, c: 0.5 * self.q[i] * off(d, i, c) ** 2) for d in range(3)] +
            [sums(lambda i, c: self.q[i] * off(d, i, c) * off(e, i, c)) for d, e in ((0, 1), (1, 2), (2, 0))])

    def tiles(self, most):
        """(first particle, count) of the cells of at most `most` particles below larger ones."""
        parent = torch.full((self.cells,), -1, device=self.p.device)
        many = torch.nonzero(self.nch > 0).flatten()
        c = torch.repeat_interleave(self.first[many] - torch.cumsum(self.nch[many], 0) + self.nch[many],
                                    self.nch[many]) + torch.arange(int(self.nch[many].sum()), device=self.p.device)
        parent[c] = torch.repeat_interleave(many, self.nch[many])
        big = torch.where(parent >= 0, self.count[parent.clamp_min(0)] > most, True)
        t = torch.nonzero((self.count <= most) & big).flatten()
        t = t[torch.argsort(self.start[t])]
        return self.start[t], self.count[t]


def _field(tab, d, eps2):
    """phi and E of charge, dipole and quadrupole (rows of tab: q, 3, 6) at offset d."""
    q, px, py, pz, xx, yy, zz, xy, yz, zx = tab
    dx, dy, dz = d
    r2 = dx * dx + dy * dy + dz * dz + eps2
    r1 = 1.0 / torch.sqrt(r2)
    i2 = r1 * r1
    r3, r5 = r1 * i2, r1 * i2 * i2
    mx, my, mz = xx * dx + 0.5 * (xy * dy + zx * dz), yy * dy + 0.5 * (xy * dx + yz * dz), zz * dz + 0.5 * (yz * dy + zx * dx)
    pd, dm, tr = px * dx + py * dy + pz * dz, dx * mx + dy * my + dz * mz, xx + yy + zz
    phi = q * r1 - pd * r3 + 3.0 * dm * r5 - tr * r3
    c = q * r3 - 3.0 * (pd + tr) * r5 + 15.0 * dm * r5 * i2
    return phi, [c * dv + pv * r3 - 6.0 * mv * r5 for dv, pv, mv in ((dx, px, mx), (dy, py, my), (dz, pz, mz))]


def _walk(tree, t, groups, theta, boxes, visit, chunk):
    """Lists of the target groups (index table, -1 pads) over all boxes; visit gets every
    accepted (cell, group): cells, targets, padding mask, offsets, leaf flags and the box."""
    th2 = theta * theta
    coc, bl2, first, nch = tree.coc.detach(), tree.bl2, tree.first, tree.nch
    most = max(1, chunk // groups.shape[1])
    for box in boxes:
        g0 = torch.arange(groups.shape[0], device=t.device)
        pend = [(g0, torch.zeros_like(g0))]
        while pend:
            g, u = pend.pop()
            if g.numel() > most:
                h = g.numel() // 2
                pend += [(g[:h], u[:h]), (g[h:], u[h:])]
                continue
            ti = groups[g]
            there = ti >= 0
            ti = ti.clamp_min(0)
            d = [(t[k][ti] - box[k]) - coc[k][u][:, None] for k in range(3)]
            ok = ((th2 * (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) > bl2[u][:, None]) | ~there).all(1)
            leaf = nch[u] == 0
            sel = torch.nonzero(ok | leaf).flatten()
            if sel.numel():
                visit(u[sel], ti[sel], there[sel], [v[sel] for v in d], leaf[sel], box)
            o = torch.nonzero(~(ok | leaf)).flatten()
            if o.numel():
                k = nch[u[o]]
                base = first[u[o]] - torch.cumsum(k, 0) + k
                pend.append((torch.repeat_interleave(g[o], k),
                             torch.repeat_interleave(base, k) + torch.arange(int(k.sum()), device=t.device)))


def _groups(case, tree, nt, dev):
    size = MODES[case["mode"]][2]
    if size == 0:
        st, cnt = tree.tiles(16)
        i = torch.arange(16, device=dev)
        return torch.where(i < cnt[:, None], st[:, None] + i, -1)
    i = torch.arange(-(-nt // size) * size, device=dev)
    return torch.where(i < nt, i, -1).reshape(-1, size)


def exact(case, seed):
    if case["n"] > NO_EXACT_ABOVE:
        return None
    dev = torch.device("cuda")
    x, y, z, q = _particles(case, seed)
    p = torch.stack([x, y, z])
    back = case["kind"] in ("fit", "grad")
    if back:
        p.requires_grad_()
        q.requires_grad_()
    tree = _Tree(p, q)
    t = tree.p.detach()
    if case["kind"] == "fit":
        t, measured = _loss(case, seed)
    eps2, ions = _eps2(case), case.get("dist") == "ions"
    tab = torch.cat([tree.coc, tree.charge[None], tree.dip, tree.quad])
    cells = tab.detach()
    out = torch.zeros((5, t.shape[1]), dtype=torch.float64, device=dev)
    groups = _groups(case, tree, t.shape[1], dev)
    near = (-1.0, 0.0, 1.0) if ions else (0.0,)
    boxes = [(i, j, k) for i in near for j in near for k in near]

    def use_of(there, d, leaf):  # not a padded slot, not the target's own leaf
        return there & ~(leaf[:, None] & (d[0] == 0) & (d[1] == 0) & (d[2] == 0))

    def add(u, ti, there, d, leaf, box):
        use = use_of(there, d, leaf)
        phi, e = _field(cells[3:, u][:, :, None], [torch.where(use, v, 1.0) for v in d], eps2)
        for k, v in enumerate((*e, phi)):
            out[k].index_add_(0, ti.flatten(), torch.where(use, v, 0.0).flatten())
        out[4].index_add_(0, ti.flatten(), there.to(torch.float64).flatten())

    _walk(tree, t, groups, case["theta"], boxes, add, 4_000_000)
    if ions:
        e, phi = _far_lattice(tree.p, tree.q, t)
        out[:3] += e
        out[3] += phi
    if case["kind"] == "host":
        r = dict(zip(("ex", "ey", "ez", "pot", "work"), out.cpu().numpy()))
        return dict(r, key=None, perm=tree.perm.cpu().numpy())
    res = dict(e=out[:3], pot=out[3], work=out[4])
    if not back:
        return res
    ge, gphi = (None, 2.0 * (out[3] - measured)) if case["kind"] == "fit" else _loss(case, seed)
    leaves = cells.clone().requires_grad_()

    def back_add(u, ti, there, d, leaf, box):
        use = use_of(there, d, leaf)
        c = leaves[:, u][:, :, None]
        phi, e = _field(c[3:], [torch.where(use, (t[k][ti] - box[k]) - c[k], 1.0) for k in range(3)], eps2)
        val = gphi[ti] * phi
        if ge is not None:
            val = val + ge[0][ti] * e[0] + ge[1][ti] * e[1] + ge[2][ti] * e[2]
        torch.where(use, val, 0.0).sum().backward()

    _walk(tree, t, groups, case["theta"], boxes, back_add, 1_000_000)
    dp, dq = torch.autograd.grad(tab, (p, q), leaves.grad)
    if case["kind"] == "fit":
        return dict(pot=res["pot"], work=res["work"], dq=dq, dx=dp)
    return dict(e=res["e"], pot=res["pot"], dq=dq, dx=dp)


# The far-lattice term of the unit cube with one layer of image boxes: the central box's
# regular expansion (order 20) through the lattice coefficients to a local expansion.
_LM = 20


def _signed(a):
    """Orders m = 0 .. L of a (L + 1, L + 1, ...) table extended to m = -L .. L."""
    m = np.arange(a.shape[1] - 1, 0, -1)
    neg = np.conj(a[:, :0:-1]) * ((-1.0) ** m).reshape((1, -1) + (1,) * (a.ndim - 2))
    return np.concatenate([neg, a], axis=1)


def _regular(lmax, x, y, z, xp=np):
    """r^l P_lm e^{-im phi} / (l + m)! by recurrence: rows (l, m >= 0)."""
    r2 = x * x + y * y + z * z
    xy = x - 1j * y
    o = {(0, 0): xp.ones_like(xy)}
    for m in range(lmax + 1):
        if m:
            o[m, m] = o[m - 1, m - 1] * xy / (2.0 * m)
        for l in range(m + 1, lmax + 1):
            v = (2.0 * l - 1.0) * z * o[l - 1, m]
            if l > m + 1:
                v = v - r2 * o[l - 2, m]
            o[l, m] = v / ((l - m) * (l + m))
    return o


def _irregular_sum(lmax, x, y, z):
    """Sum over the points of (l - m)! P_lm e^{im phi} / r^(l+1), a (l, m >= 0) table."""
    i2 = 1.0 / (x * x + y * y + z * z)
    a = np.zeros((lmax + 1, lmax + 1), complex)
    d = np.sqrt(i2) + 0j
    for m in range(lmax + 1):
        if m:
            d = d * (2.0 * m - 1.0) * (x + 1j * y) * i2
        prev, cur = np.zeros_like(d), d
        for l in range(m, lmax + 1):
            if l > m:
                prev, cur = cur, ((2.0 * l - 1.0) * z * cur - ((l - 1.0) ** 2 - m * m) * prev) * i2
            a[l, m] = cur.sum()
    return a


def _m2l(a, b):
    """sum over j, k of (-1)^j a(j + l, k + m) b(j, k) for m >= 0, a and b with signed orders."""
    la, lb = a.shape[0] - 1, b.shape[0] - 1
    big = np.zeros((la + lb + 1, 2 * (la + lb) + 1), complex)
    big[: la + 1, lb: lb + 2 * la + 1] = a
    out = np.zeros((la + 1, la + 1), complex)
    c = la + lb
    for j in range(lb + 1):
        for k in range(-j, j + 1):
            out += (-1.0) ** j * b[j, lb + k] * big[j: j + la + 1, c + k: c + k + la + 1]
    return np.tril(out)


@functools.lru_cache(maxsize=1)
def _lattice():
    lm, lt = 50, 100  # the unit cube's coefficients are those of order 50
    near = np.array([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)], float)
    o = _regular(lm, *(-near.T))
    ms = np.zeros((lm + 1, lm + 1), complex)
    for (l, m), v in o.items():
        ms[l, m] = v.sum()
    far = 3.0 * near[np.abs(near).sum(1) > 0][:, None, :] + near[None]
    ls = _irregular_sum(lt, *far.reshape(-1, 3).T)
    ms, scale = _signed(ms), 3.0 ** -(np.arange(lt + 1.0) + 1.0)
    ml = ls
    for _ in range(32):
        ml = _m2l(_signed(ml * scale[:, None]), ms) + ls
    keep = np.zeros((2 * _LM + 1, 2 * _LM + 1))
    keep[::2, ::4] = 1.0  # the cube's symmetry
    return np.tril(ml.real[: 2 * _LM + 1, : 2 * _LM + 1] * keep) + 0j


def _far_lattice(p, q, t):
    """E and phi of everything beyond the image boxes, net dipole cancelled by charges at the corners."""
    dip = ((p - 0.5) * q).sum(1)
    corner = torch.cat([torch.eye(3, dtype=p.dtype, device=p.device), torch.zeros((3, 1), dtype=p.dtype, device=p.device)], 1)
    cq = torch.cat([-dip, dip.sum()[None]])
    om = np.zeros((_LM + 1, _LM + 1), complex)
    for (l, m), v in _regular(_LM, *(torch.cat([p, corner], 1) - 0.5), xp=torch).items():
        om[l, m] = complex((v * torch.cat([q, cq])).sum())
    om[0, 0] = 0.0
    mu = _signed(_m2l(_signed(_lattice()), _signed(om))[: _LM + 2, : _LM + 2])
    mu[_LM + 1] = 0.0
    c = _LM + 1
    phi = torch.zeros_like(t[0])
    e = torch.zeros_like(t)
    for (a, b), v in _regular(_LM, *(t - 0.5), xp=torch).items():
        for s in ((1, -1) if b else (1,)):
            o = v if s == 1 else (-1.0) ** b * v.conj()
            if a <= _LM:
                phi += (o * complex(mu[a, c + s * b])).real
            if a < _LM:
                w = o * complex(mu[a + 1, c + s * b + 1])
                e[0] -= w.real
                e[1] -= w.imag
                e[2] -= (o * complex(mu[a + 1, c + s * b])).real
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                for f in range(4):
                    d = t - torch.tensor([i, j, k], dtype=t.dtype, device=t.device)[:, None] - corner[:, f: f + 1]
                    r = cq[f] / d.norm(dim=0)
                    phi += r
                    e += d * (r / (d * d).sum(0))
    return e, phi
