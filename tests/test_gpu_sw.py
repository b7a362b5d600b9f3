"""The hooking Swendsen-Wang kernel: site and bond counts around its words of 32
bits and quads of bonds, fields (bonds to the dummy spin), isolated sites, both
launch shapes, couplings of every strength."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sparse(n, bonds, rng, field):
    a, b = rng.integers(0, n, bonds), rng.integers(0, n, bonds)
    keep = a != b
    a, b = a[keep], b[keep]
    h = rng.uniform(-1, 1, n) * (rng.random(n) < field)
    return I.augmented_from_ising(h, (np.minimum(a, b), np.maximum(a, b), rng.normal(size=a.size)), n)


@pytest.mark.parametrize("n,bonds,field,R", [(1024, 2000, 0.5, 3), (1055, 1, 0.0, 2), (1055, 4001, 0.0, 40),
                                             (1311, 3303, 1.0, 148), (2048, 9000, 0.01, 5), (8192, 16001, 0.3, 3),
                                             (8223, 20000, 0.0, 170)])
def test_swendsen_wang_hooking_bit_exact(ctx, n, bonds, field, R):
    rng = np.random.default_rng(n + bonds)
    g = O.AugCSR(_sparse(n, bonds, rng, field))
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    betas = np.array([0.05, 0.4, 1.5, 6.0])
    mcs = np.ones(4, np.int32)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, n))
    s = s0.copy()
    N.sw_run(dg, s, betas, mcs, seed=61, replica_offset=32)
    padded = np.concatenate([np.ones((32, n), np.int8), s0])
    np.testing.assert_array_equal(s, O.replay_sw(g, padded, betas.astype(np.float32), 61)[32:])


def test_swendsen_wang_hooking_lattice_bit_exact(ctx):
    g = O.AugCSR(I.lattice_pm_j(64, seed=3)[0])
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    betas, mcs = I.geometric_betas(0.1, 5.0, 8)
    s0 = np.random.default_rng(1).choice(np.array([-1, 1], np.int8), size=(6, g.n))
    s = s0.copy()
    st = N.sw_run(dg, s, betas, mcs, seed=62)
    np.testing.assert_array_equal(s, O.replay_sw(g, s0, np.repeat(betas, mcs).astype(np.float32), 62))
    assert st["threads"] == 1024


@pytest.mark.parametrize("side", [212, 214, 216, 218])
def test_swendsen_wang_around_the_shared_memory_limits_bit_exact(ctx, side):
    """Sides on either side of both kernels' shared-memory limits; only the last
    keeps its links in global scratch."""
    g = O.AugCSR(I.lattice_pm_j(side, seed=4)[0])
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    betas = np.array([0.3, 2.0])
    s0 = np.random.default_rng(side).choice(np.array([-1, 1], np.int8), size=(2, g.n))
    s = s0.copy()
    N.sw_run(dg, s, betas, np.ones(2, np.int32), seed=63)
    np.testing.assert_array_equal(s, O.replay_sw(g, s0, betas.astype(np.float32), 63))


@pytest.mark.parametrize("n,bonds,field,R", [(1055, 2100, 0.0, 2), (2055, 6700, 0.0, 149), (8223, 20000, 0.3, 170),
                                             (8192, 9000, 0.0, 300), (46015, 1, 0.0, 2)])
def test_swendsen_wang_hooking_near_neighbours_bit_exact(ctx, n, bonds, field, R):
    """Bonds between sites of near indices, which the hooking kernel takes with
    several replicas an SM too."""
    rng = np.random.default_rng(n + bonds)
    pair = rng.choice((n - 60) * 60, bonds, replace=False)
    a, b = pair // 60, pair // 60 + pair % 60 + 1
    h = rng.uniform(-1, 1, n) * (rng.random(n) < field)
    g = O.AugCSR(I.augmented_from_ising(h, (a, b, rng.normal(size=bonds)), n))
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    betas = np.array([0.4, 1.5])
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, n))
    s = s0.copy()
    N.sw_run(dg, s, betas, np.ones(2, np.int32), seed=64)
    np.testing.assert_array_equal(s, O.replay_sw(g, s0, betas.astype(np.float32), 64))
