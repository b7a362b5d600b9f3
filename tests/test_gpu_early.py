"""Sweep and field kernels that follow one another start early (their set-up runs
while the kernel before finishes, and the field kernel zeroes the sweep kernel's item
counter): every segment must still see the finished spins and fields of the one before,
launched directly or replayed as a graph."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# odd sizes (rows that share lines and are copied byte by byte), fewer and more
# work items than the device holds, shared-memory and global couplings, and a
# last segment of one sweep
@pytest.mark.parametrize("sizes,reads,sweeps", [((129,), 1, 49), ((151, 130), 37, 33), ((777,), 9, 40),
                                                ((150, 260, 133), 3000, 18)])
@pytest.mark.parametrize("graph", ["1", "0"])
def test_early_segments_bit_exact(ctx, monkeypatch, sizes, reads, sweeps, graph):
    monkeypatch.setenv("OJ_GRAPH", graph)
    mats = [I.dense_qubo_normal(n, seed=500 + k)[0].toarray() for k, n in enumerate(sizes)]
    betas, mcs = I.geometric_betas(0.1, 6.0, sweeps)
    counts = [reads] * len(sizes)
    s0 = np.random.default_rng(sweeps).choice(np.array([-1, 1], np.int8), size=reads * sum(sizes))
    s = s0.copy()
    st = N.sa_run_batched(N.Batch(ctx, mats), counts, s, betas, mcs, seed=19)
    want, drift = O.replay_sa_batch(mats, counts, s0, np.repeat(betas, mcs).astype(np.float32), 19, drift=True)
    np.testing.assert_array_equal(s, want)
    assert st["field_drift"] == drift.max()
