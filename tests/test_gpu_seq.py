"""Small dense graphs through the colour-class kernels' serial path: sizes at
the edges of its groups of four sites, blocks of sixteen and last tree, replica
counts from one tree per warp to one lane per chain, every kind of slice count."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _instance(n, density, seed):
    rng = np.random.default_rng(seed)
    J = np.triu(rng.uniform(-1, 1, (n, n)) * (rng.random((n, n)) < density), 1)
    g = O.AugCSR(I.dense_augmented(J + J.T, rng.uniform(-1, 1, n)))
    return g, rng


@pytest.mark.parametrize("n,density", [(1, 1.0), (2, 1.0), (5, 1.0), (6, 0.7), (16, 1.0), (17, 0.5), (33, 1.0),
                                       (64, 1.0), (97, 0.5), (176, 1.0)])
@pytest.mark.parametrize("R", [1, 31, 1500, 5000])
def test_sa_serial_path_bit_exact(ctx, n, density, R):
    if n > 64 and R > 1500:
        R = 2500
    g, rng = _instance(n, density, n)
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    betas, mcs = I.geometric_betas(0.1, 5.0, 4)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, n))
    s = s0.copy()
    st = N.sa_run(dg, s, betas, mcs, seed=31, kernel="colour", replica_offset=64)
    ref = O.replay_sa(g, s0, np.repeat(betas, mcs).astype(np.float32), 31, mode="colour", rep0=64)
    np.testing.assert_array_equal(s, ref)
    assert st["kernel"] == "colour"


@pytest.mark.parametrize("n,density", [(2, 1.0), (7, 1.0), (20, 0.6), (65, 1.0), (130, 1.0)])
@pytest.mark.parametrize("T,R", [(2, 3), (3, 200), (4, 700), (7, 40), (16, 33), (33, 5), (64, 3), (4, 3000)])
def test_sqa_serial_path_bit_exact(ctx, n, density, T, R):
    if n > 64 and R > 700:
        R = 1000
    g, rng = _instance(n, density, n + T)
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    ss = np.array([0.0, 0.4, 1.0])
    betas, mcs = np.full(3, 4.0), np.ones(3, np.int32)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, T, n))
    s = s0.copy()
    N.sqa_run(dg, s, 1.0, betas, ss, mcs, seed=32, kernel="colour")
    a, b = O.sqa_coefficients(betas, ss, 1.0, T)
    np.testing.assert_array_equal(s, O.replay_sqa(g, s0, a, b, 32))
