"""GPU: the far-lattice step and force at particle counts around their work
split (two particles per warp, 16 warps per block, 148 blocks), target counts
around the force's blocks, and each set of periodic directions, against the oracle.

Tolerance 1e-11 of the field's scale: both sides are FP64 sums over the same
orders, the particle sums in different orders of some thousand terms."""
import os

import numpy as np
import pytest

import pepc_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "reference_pins.npz"))


def check(n, nt, seed, **kw):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random(n), rng.random(n), rng.random(n)
    q = rng.standard_normal(n)
    kw = dict(theta2=0.16, eps2=0.0, **kw)
    cube = all(kw["periodicity"])
    if not cube:  # a cell without a table: coefficients by the iteration on both sides
        kw.update(t_lattice_1=(1.25, 0.0, 0.0))
    tc, orc = P.TreeCode(**kw), O.Oracle(num_threads=8, **kw)
    if cube:
        orc.set_lattice_coefficients(O.reference_lattice_table(GOLD))
    tc.pepc_grow_tree(x, y, z, q)
    orc.grow_tree(x, y, z, q)
    # away from the corners, where the reference's fictitious charges (1e-16 of
    # q / r^2 each) cancel only to their rounding
    t = 0.05 + 0.9 * rng.random((3, nt))
    a, b = tc.lattice(*t), orc.lattice(*t)
    for k in ("ex", "ey", "ez", "pot"):
        assert np.abs(a[k] - b[k]).max() <= 1e-11 * np.abs(b[k]).max(), (n, nt, k)
    tc.close()
    orc.close()


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 1023, 148 * 32 - 1, 148 * 32 + 1, 20011])
def test_particle_counts(gpu, n):
    check(n, 70, 5, periodicity=(1, 1, 1))


@pytest.mark.parametrize("nt", [1, 127, 128, 129, 148 * 6 * 128 + 1])
def test_target_counts(gpu, nt):
    check(50, nt, 6, periodicity=(1, 1, 1))


@pytest.mark.parametrize("corr", [0, 1, 2])
@pytest.mark.parametrize("per", [(1, 0, 0), (0, 1, 1), (1, 1, 1)])
def test_periodic_directions(gpu, per, corr):
    check(400, 200, 7, periodicity=per, fmm_extrinsic_correction=corr)


def test_two_layers_of_boxes(gpu):
    # no table for two layers: in one direction, where the iteration has no
    # conditionally convergent entries
    check(400, 200, 8, periodicity=(1, 0, 0), mirror_box_layers=2)
