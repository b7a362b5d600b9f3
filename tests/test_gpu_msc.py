"""The bit-packed SA kernel's forms: one CTA per group without cluster barriers,
clusters, draws side by side or one by one, at class sizes around the thread
counts and for every degree."""
import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [("lattice", 5), ("lattice", 8), ("lattice", 26), ("lattice", 35), ("lattice", 37),
                                   ("lattice", 47), ("regular", 40, 1), ("regular", 600, 3), ("regular", 300, 5),
                                   ("regular", 200, 8)])
@pytest.mark.parametrize("shape", [None, (1, 64), (1, 1024), (2, 256), (3, 512)])
def test_bitpacked_forms_bit_exact(ctx, monkeypatch, which, shape):
    m, _ = I.lattice_pm_j(which[1], seed=9) if which[0] == "lattice" else I.random_regular_pm_j(which[1], which[2],
                                                                                               seed=9, max_tries=10**5) \
        if which[2] < 5 else _circulant(which[1], which[2])
    g = O.AugCSR(m)
    if shape is not None:
        monkeypatch.setenv("OJ_MSC_CLUSTER", str(shape[0]))
        monkeypatch.setenv("OJ_MSC_THREADS", str(shape[1]))
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    info = dg.info()
    betas, mcs = I.geometric_betas(0.05, 4.0, 12)
    rng = np.random.default_rng(which[1])
    for R in (1, 70):
        s0 = rng.choice(np.array([-1, 1], np.int8), size=(R, g.n))
        s = s0.copy()
        st = N.sa_run(dg, s, betas, mcs, seed=51, kernel="bitpacked")
        if shape is not None:
            assert (st["cluster"], st["threads"]) == shape
        thr, alw = O.msc_thresholds(np.repeat(betas, mcs).astype(np.float32), info["coupling_abs"], info["max_degree"])
        padded = np.ones(((R + 31) // 32 * 32, g.n), np.int8)
        padded[:R] = s0
        np.testing.assert_array_equal(s, O.replay_sa_msc(g, padded, thr, alw, 51)[:R])


def _circulant(n, d):
    """Regular graph of degree d: i couples to i +- 1 .. i +- d // 2, and for odd d
    to the opposite site."""
    rng = np.random.default_rng(d)
    pairs = {(min(i, (i + k) % n), max(i, (i + k) % n)) for i in range(n) for k in range(1, d // 2 + 1)}
    if d % 2:
        pairs |= {(i, i + n // 2) for i in range(n // 2)}
    a, b = np.array(sorted(pairs)).T
    return I.augmented_from_ising(np.zeros(n), (a, b, rng.choice([-1.0, 1.0], size=a.size)), n), 0.0


@pytest.mark.parametrize("which", [(40, 1), (70, 2), (130, 3), (1000, 3), (4200, 3), (300, 4), (200, 5), (96, 6),
                                   (98, 7), (120, 8)])
@pytest.mark.parametrize("T,R", [(2, 40), (8, 5), (32, 3), (64, 2)])
def test_slice_split_forms_bit_exact(ctx, which, T, R):
    """The slice-split SQA kernel's default shapes: one CTA per group and clusters,
    tables written a sweep ahead or at the sweep's start, every degree."""
    n, d = which
    m, _ = I.random_regular_pm_j(n, d, seed=9, max_tries=10**5) if d < 4 else _circulant(n, d)
    g = O.AugCSR(m)
    dg = N.Graph(ctx, g.n, g.indptr, g.indices, g.data)
    info = dg.info()
    ss = np.array([0.0, 0.2, 0.6, 0.9, 1.0])
    betas, mcs = np.full(5, 4.0), np.ones(5, np.int32)
    s0 = np.random.default_rng(n + T).choice(np.array([-1, 1], np.int8), size=(R, T, n))
    s = s0.copy()
    st = N.sqa_run(dg, s, 1.0, betas, ss, mcs, seed=52, kernel="bitpacked")
    a, b = O.sqa_coefficients(betas, ss, 1.0, T)
    thr, mode = O.sqa_msc_thresholds(a, b, info["coupling_abs"], info["max_degree"])
    np.testing.assert_array_equal(s, O.replay_sqa_split(g, s0, thr, mode, 52))
    assert (st["cluster"] > 1) == (n == 4200 and R <= 8 * max(1, 32 // (T // 2)))
