"""The colour-class kernels at the edge of shared memory: the largest spins that
fit it, the smallest that do not, and graphs whose tables cannot be allocated;
the kernels on either side give the same spins."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cycle(n):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    j = (i + 1) % n
    m = I.augmented_from_ising(rng.uniform(-1, 1, n), (np.minimum(i, j), np.maximum(i, j), rng.uniform(-1, 1, n)), n)
    return O.AugCSR(m), rng


def _check_sa(ctx, g, dg, rng, R):
    betas, mcs = I.geometric_betas(0.1, 3.0, 3)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, g.n))
    s = s0.copy()
    N.sa_run(dg, s, betas, mcs, seed=51, kernel="colour")
    np.testing.assert_array_equal(s, O.replay_sa(g, s0, np.repeat(betas, mcs).astype(np.float32), 51, mode="colour"))


def _check_sqa(ctx, g, dg, rng, T, R):
    ss, betas, mcs = np.array([0.2, 0.8]), np.full(2, 4.0), np.ones(2, np.int32)
    s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, T, g.n))
    s = s0.copy()
    N.sqa_run(dg, s, 1.0, betas, ss, mcs, seed=52, kernel="colour")
    a, b = O.sqa_coefficients(betas, ss, 1.0, T)
    np.testing.assert_array_equal(s, O.replay_sqa(g, s0, a, b, 52))


@pytest.mark.parametrize("n,R", [(51201, 9), (204800, 2), (204801, 5)])
def test_sa_colour_at_the_shared_memory_limit(ctx, n, R):
    g, rng = _cycle(n)
    _check_sa(ctx, g, N.Graph(ctx, g.n, g.indptr, g.indices, g.data), rng, R)


@pytest.mark.parametrize("n,T", [(102400, 9), (102401, 16), (68266, 17), (68267, 17)])
def test_sqa_colour_at_the_shared_memory_limit(ctx, n, T):
    g, rng = _cycle(n)
    _check_sqa(ctx, g, N.Graph(ctx, g.n, g.indptr, g.indices, g.data), rng, T, 2)


def test_colour_runs_without_room_for_the_tables():
    g, rng = _cycle(3001)
    for check in (lambda c, dg: _check_sa(c, g, dg, rng, 6), lambda c, dg: _check_sqa(c, g, dg, rng, 5, 3)):
        failed = 0
        for k in range(20):
            ctx = N.Context(0)
            dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
            ctx.inject_alloc_failure(k)
            try:
                check(ctx, dg)
            except N.OJError as err:  # a buffer of the call itself
                assert err.status == N.OJ_ERR_OOM
                failed += 1
            ctx.inject_alloc_failure(None)
            check(ctx, dg)
            ctx.close()
        assert 0 < failed < 19
