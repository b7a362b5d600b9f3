"""One-chunk batches (instances of at most 128 sites): the recompute's grid integers
from shared memory (a CTA per SM) and from global memory (more work items than SMs),
and both default launch shapes."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,reads", [((1, 7, 128), 3), ((100,), 100), ((33, 97, 128, 64) * 11, 16),
                                         ((20, 120), 700)])
def test_one_chunk_recompute_bit_exact(ctx, sizes, reads):
    mats = [I.dense_qubo_normal(n, seed=300 + k)[0].toarray() for k, n in enumerate(sizes)]
    betas, mcs = I.geometric_betas(0.1, 4.0, 37)
    total = reads * sum(sizes)
    s0 = np.random.default_rng(len(sizes)).choice(np.array([-1, 1], np.int8), size=total)
    s = s0.copy()
    counts = [reads] * len(sizes)
    st = N.sa_run_batched(N.Batch(ctx, mats), counts, s, betas, mcs, seed=71)
    assert st["variant"] == (45 if reads * len(sizes) <= 1184 else 83)
    np.testing.assert_array_equal(s, O.replay_sa_batch(mats, counts, s0, np.repeat(betas, mcs).astype(np.float32), 71))
