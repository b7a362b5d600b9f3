"""The colour-class kernels with the spins in shared memory: classes at the
edges of a slice of 32 sites, lists from empty to long, replica counts from one
partial group to several CTAs per SM, slice counts at the edges of an octet."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cycle(n, rng):
    i = np.arange(n)
    j = (i + 1) % n
    return I.augmented_from_ising(rng.uniform(-1, 1, n), (np.minimum(i, j), np.maximum(i, j), rng.uniform(-1, 1, n)), n)


def _random(n, degree, rng):
    J = np.triu(rng.uniform(-1, 1, (n, n)) * (rng.random((n, n)) < degree / n), 1)
    return I.dense_augmented(J + J.T, rng.uniform(-1, 1, n))


def _graph(ctx, which):
    rng = np.random.default_rng(len(which) + which[1])
    m = _cycle(which[1], rng) if which[0] == "cycle" else _random(which[1], which[2], rng)
    g = O.AugCSR(m)
    return g, N.Graph(ctx, g.n, g.indptr, g.indices, g.data), rng


@pytest.mark.parametrize("which", [("cycle", 62), ("cycle", 64), ("cycle", 66), ("cycle", 131), ("random", 300, 5),
                                   ("random", 300, 90)])
@pytest.mark.parametrize("R", [1, 4, 9, 601, 1300, 5003])
def test_sa_colour_slices_and_groups_bit_exact(ctx, which, R):
    if which[-1] == 90 and R > 601:
        R = 700
    g, dg, rng = _graph(ctx, which)
    betas, mcs = I.geometric_betas(0.1, 3.0, 4)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, g.n))
    s = s0.copy()
    N.sa_run(dg, s, betas, mcs, seed=41, kernel="colour", replica_offset=32)
    ref = O.replay_sa(g, s0, np.repeat(betas, mcs).astype(np.float32), 41, mode="colour", rep0=32)
    np.testing.assert_array_equal(s, ref)


@pytest.mark.parametrize("which", [("cycle", 64), ("cycle", 67), ("random", 250, 4), ("random", 260, 80)])
@pytest.mark.parametrize("T,R", [(2, 5), (3, 5), (4, 700), (5, 3), (7, 3), (8, 300), (9, 3), (16, 4), (17, 3), (66, 2)])
def test_sqa_colour_octets_bit_exact(ctx, which, T, R):
    if which[-1] == 80:
        R = min(R, 150)
    g, dg, rng = _graph(ctx, which)
    ss = np.array([0.0, 0.5, 1.0])
    betas, mcs = np.full(3, 4.0), np.ones(3, np.int32)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, T, g.n))
    s = s0.copy()
    N.sqa_run(dg, s, 1.0, betas, ss, mcs, seed=42, kernel="colour")
    a, b = O.sqa_coefficients(betas, ss, 1.0, T)
    np.testing.assert_array_equal(s, O.replay_sqa(g, s0, a, b, 42))
