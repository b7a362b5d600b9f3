"""The library's host code on the CPU, its objects linked against a stand-in
for the CUDA runtime (fake/fake_cuda.cpp): the order of uploads and launches,
what device memory a call takes and gives back, which kernel a call reaches.
Kernels do not run, so spins stay as they are."""
import ctypes as C
import gc
import glob
import importlib.util
import os
import subprocess

import numpy as np
import pytest

from openjij_b200 import _native as N
from openjij_b200 import instances as I

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("_recipe", os.path.join(HERE, "..", "openjij_b200", "build.py"))
    recipe = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(recipe)
    recipe.build_cuda()
    out = str(tmp_path_factory.mktemp("fake") / "libojb200_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                    "-I" + os.path.join(os.path.dirname(recipe.NVCC), "..", "include"),
                    os.path.join(HERE, "fake", "fake_cuda.cpp")] + sorted(glob.glob(recipe.BUILD + "/*.o")) +
                   ["-o", out], check=True)
    return out


@pytest.fixture
def fake(fake_lib):
    """The library on the stand-in, in place of the real one; its context is fake.ctx."""
    saved = N._lib, N.LIB_PATH
    N._lib, N.LIB_PATH = None, fake_lib
    lib = N.lib()
    for name in ("fake_live_bytes", "fake_peak_bytes"):
        getattr(lib, name).restype = C.c_size_t
    lib.fake_launches.restype = C.c_char_p
    lib.fake_fail_new.argtypes = [C.c_longlong, C.c_size_t]
    lib.ctx = N.Context(0)
    lib.fake_reset()
    yield lib
    lib.ctx.close()
    gc.collect()
    N._lib, N.LIB_PATH = saved


def _chimera(ctx, cells, seed=1):
    return N.Graph(ctx, *I.augmented_csr(I.chimera_pm_j(cells, seed=seed, field=0.5)[0]))


def _lattice(ctx, side, seed=1):
    return N.Graph(ctx, *I.augmented_csr(I.lattice_pm_j(side, seed=seed)[0]))


def _first_sa(ctx, kernel, make):
    g = make(ctx)
    N.sa_run(g, np.ones((3, g.n), np.int8), [1.0], [2], seed=1, kernel=kernel, energies=np.zeros(3))


def _first_sqa(ctx, kernel, make, T):
    g = make(ctx)
    N.sqa_run(g, np.ones((3, T, g.n), np.int8), 1.0, [1.0], [0.5], [2], seed=1, kernel=kernel)


def _first_sw(ctx, make):
    g = make(ctx)
    N.sw_run(g, np.ones((3, g.n), np.int8), [1.0], [2], seed=1)


def _first_batch(ctx):
    mats = [I.dense_qubo_normal(n, seed=n)[0].toarray() for n in (40, 200)]
    N.sa_run_batched(N.Batch(ctx, mats), [2, 3], np.ones(2 * 40 + 3 * 200, np.int8), [1.0], [2], seed=1)


def _dense(ctx):
    return N.Graph(ctx, *I.augmented_csr(I.dense_ising_uniform(90, seed=1)[0]))


@pytest.mark.parametrize("call", [
    lambda ctx: _first_sa(ctx, "colour", lambda c: _chimera(c, 6)),
    lambda ctx: _first_sqa(ctx, "colour", lambda c: _chimera(c, 6), 5),
    lambda ctx: _first_sa(ctx, "bitpacked", lambda c: _lattice(c, 16)),
    lambda ctx: _first_sqa(ctx, "bitpacked", lambda c: _lattice(c, 16), 8),
    lambda ctx: _first_sqa(ctx, "bitpacked", lambda c: _lattice(c, 16), 7),
    lambda ctx: _first_sw(ctx, lambda c: _lattice(c, 40)),
    lambda ctx: _first_sw(ctx, lambda c: _chimera(c, 4)),
    lambda ctx: _first_sa(ctx, "dense_jump", _dense),
    lambda ctx: _first_sa(ctx, "dense_plain", _dense),
    lambda ctx: _first_sa(ctx, "dense_tc", _dense),
    _first_batch,
], ids=["sa colour", "sqa colour", "sa bit-packed", "sqa slice-split", "sqa bit-packed", "sw hooking", "sw",
        "dense jump", "dense plain", "dense tc", "batch"])
def test_tables_are_on_the_device_before_the_first_launch(fake, call):
    """A graph's or batch's tables are uploaded by copies that may return
    before the data is on the device; the context's stream does not wait for
    them by itself."""
    call(fake.ctx)
    assert fake.fake_launches()
    assert fake.fake_unordered() == 0


def test_a_failing_host_allocation_of_the_colour_tables_leaks_no_device_memory(fake):
    """Every host allocation of the first run's table build fails in turn: the
    run is out of memory, the graph is usable, and destroying both gives all
    device memory back."""
    n = 40000
    i = np.arange(n)
    m = I.augmented_from_ising(np.full(n, 0.25), (np.minimum(i, (i + 1) % n), np.maximum(i, (i + 1) % n), i % 7 + 1.0), n)
    aug = I.augmented_csr(m)
    fake.ctx.close()
    for k in range(100):
        before = fake.fake_live_bytes()
        ctx = N.Context(0)
        g = N.Graph(ctx, *aug)
        s = np.ones((1, n), np.int8)
        fake.fake_fail_new(k, 64 * 1024)
        try:
            N.sa_run(g, s, [1.0], [1], seed=1, kernel="colour")
        except N.OJError as err:
            assert err.status == N.OJ_ERR_OOM
        done = fake.fake_new_pending()
        fake.fake_fail_new(-1, 0)
        N.sa_run(g, s, [1.0], [1], seed=1, kernel="colour")
        g.close()
        ctx.close()
        if k > 0:  # the first context sets up what the process keeps
            assert fake.fake_live_bytes() == before, k
        if done:
            break
    assert 0 < k < 99


def test_plans_of_several_cluster_sizes_are_bounded_and_given_back(fake):
    """The number of replicas sets the cluster size of the bit-packed kernel;
    calls that alternate it build each size's plan once."""
    fake.ctx.close()
    ctx = N.Context(0)
    before = fake.fake_live_bytes()
    g = _lattice(ctx, 72)
    sizes = set()
    for turn in range(3):
        for R in (32, 640, 1600):
            sizes.add(N.sa_run(g, np.ones((R, g.n), np.int8), [1.0], [1], seed=1, kernel="bitpacked")["cluster"])
        live = fake.fake_live_bytes()
        assert turn == 0 or live == first
        first = live
    assert len(sizes) > 1
    g.close()
    ctx.close()
    assert fake.fake_live_bytes() <= before


def test_a_context_gives_back_its_buffers(fake):
    fake.ctx.close()
    before = fake.fake_live_bytes()
    ctx = N.Context(0)
    g = _dense(ctx)
    b = N.Batch(ctx, [I.dense_qubo_int(200, seed=1)[0].toarray()])
    N.sa_run(g, np.ones((3, g.n), np.int8), [1.0], [2], seed=1, energies=np.zeros(3))
    N.sa_run_batched(b, [40], np.ones(40 * 200, np.int8), [1.0], [2], seed=1, energies=np.zeros(40))
    N.sqa_run(g, np.ones((3, 4, g.n), np.int8), 1.0, [1.0], [0.5], [2], seed=1, energies=np.zeros((3, 4)))
    b.close()
    g.close()
    ctx.close()
    assert fake.fake_live_bytes() <= before


@pytest.mark.parametrize("failing", ["device", "host"])
def test_a_colour_run_without_room_for_its_tables_reads_the_neighbour_lists(fake, failing):
    """The tables of the shared-memory colour kernels are only there for speed:
    where they cannot be allocated, the run takes the kernels that read the
    graph's own lists, as one too large for shared memory does."""
    n = 40000
    i = np.arange(n)
    m = I.augmented_from_ising(np.full(n, 0.25), (np.minimum(i, (i + 1) % n), np.maximum(i, (i + 1) % n), i % 7 + 1.0), n)
    g = N.Graph(fake.ctx, *I.augmented_csr(m))
    s = np.ones((1, 3, n), np.int8)

    def sa():
        N.sa_run(g, s[:, 0], [1.0], [1], seed=1, kernel="colour")

    def sqa():
        N.sqa_run(g, s, 1.0, [1.0], [0.5], [1], seed=1, kernel="colour")

    N.sw_run(g, s[:, 0], [1.0], [1], seed=1, energies=np.zeros(1))  # sizes the context's buffers
    fake.ctx.inject_alloc_failure(10**6)
    for run, kernel in ((sa, b"sa_colour_global_kernel"), (sqa, b"sqa_colour_global_kernel")):
        for k in range(20):
            fake.fake_reset()
            if failing == "host":
                fake.fake_fail_new(k, 64 * 1024)
            else:
                fake.ctx.inject_alloc_failure(k)
            try:
                run()
            except N.OJError as err:  # a buffer of the call itself
                assert err.status == N.OJ_ERR_OOM
            else:
                if fake.fake_launches().count(kernel):
                    break
        else:
            raise AssertionError("no failing allocation reached " + kernel.decode())
        fake.fake_fail_new(-1, 0)
        fake.ctx.inject_alloc_failure(None)
    fake.fake_reset()
    sa()  # with room again the tables are built
    assert b"global" not in fake.fake_launches()


def _circulant(ctx, n, degree, seed=1):
    """+-J couplings to the sites at degree / 2 random offsets on either side: a
    regular graph on which every part of a partition borders most others."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    a = np.tile(i, degree // 2)
    b = np.concatenate([(i + k) % n for k in rng.choice(np.arange(1, n // 2), degree // 2, replace=False)])
    m = I.augmented_from_ising(np.zeros(n), (np.minimum(a, b), np.maximum(a, b), rng.choice([-1.0, 1.0], a.size)), n)
    return N.Graph(ctx, *I.augmented_csr(m))


@pytest.mark.parametrize("n,degree,R", [(40000, 8, 400), (60000, 6, 32), (30000, 8, 400)])
def test_bitpacked_runs_take_a_cluster_that_their_partition_fits(fake, n, degree, R):
    """The number of CTAs a group gets follows the number of groups; the halos of
    a graph without locality may need more of them."""
    g = _circulant(fake.ctx, n, degree)
    st = N.sa_run(g, np.ones((R, n), np.int8), [1.0], [1], seed=1, kernel="bitpacked")
    assert st["cluster"] <= 16


def test_swendsen_wang_takes_union_find_scratch_only_for_the_kernel_that_uses_it(fake):
    """A lattice of side 214 has more sites than the walking kernel holds in
    shared memory, but the hooking kernel takes it; side 230 fits neither."""
    for side, kernel, needs in ((214, b"sw_hook_kernel", False), (230, b"sw_kernel", True)):
        g = _lattice(fake.ctx, side)
        R = 100
        fake.fake_reset()
        before = fake.fake_live_bytes()
        N.sw_run(g, np.ones((R, g.n), np.int8), [1.0], [1], seed=1)
        assert kernel in fake.fake_launches()
        forest = 4 * R * (g.n + 1)
        assert (fake.fake_live_bytes() - before >= forest) == needs
        g.close()


@pytest.mark.parametrize("sizes,reads,variant", [
    (np.linspace(100, 700, 200), 24, 45), (np.linspace(100, 700, 200), 32, 83),
    (np.linspace(64, 1024, 512), 12, 45), (np.linspace(64, 1024, 512), 16, 83),
    ([777], 2960, 45), ([777], 2961, 83), ([777], 3553, 45), ([1300], 2048, 83), ([1300], 1776, 45),
    ([2048], 4096, 45), ([512], 4096, 83)])
def test_default_variant_of_large_instances(fake, sizes, reads, variant):
    """More than 512 sites: the variant with more loads in flight, except where
    the one with more replicas an SM runs them in fewer turns."""
    sizes = np.asarray(sizes, int)
    b = N.Batch(fake.ctx, [np.pad([[1.0]], ((n, 0), (n, 0))) for n in sizes])
    st = N.sa_run_batched(b, np.full(len(sizes), reads, np.int32), np.ones(int(sizes.sum()) * reads, np.int8), [1.0],
                          [1], seed=1)
    assert st["variant"] == variant
    if len(sizes) == 1:
        g = N.Graph(fake.ctx, *I.augmented_csr(I.dense_qubo_int(int(sizes[0]), seed=1)[0]))
        st = N.sa_run(g, np.ones((reads, g.n), np.int8), [1.0], [1], seed=1, kernel="dense_jump")
        assert st["variant"] == variant


def _lattice_shuffled(ctx, side):
    m = I.lattice_pm_j(side, seed=1)[0].tocoo()
    n = side * side
    to = np.append(np.random.default_rng(1).permutation(n), n)
    m.row, m.col = to[m.row], to[m.col]
    return N.Graph(ctx, *I.augmented_csr(m.tocsr()))


@pytest.mark.parametrize("make,R,hooks", [
    (lambda c: _lattice(c, 32), 148, False), (lambda c: _lattice(c, 33), 148, True), (lambda c: _lattice(c, 33), 149, False),
    (lambda c: _lattice(c, 56), 256, False), (lambda c: _lattice(c, 64), 296, True), (lambda c: _lattice(c, 64), 297, False),
    (lambda c: _lattice(c, 91), 1024, True), (lambda c: _lattice_shuffled(c, 91), 148, True),
    (lambda c: _lattice_shuffled(c, 91), 149, False), (lambda c: _lattice_shuffled(c, 200), 1024, True),
    (lambda c: _lattice_shuffled(c, 214), 1024, True), (lambda c: _chimera(c, 16), 256, True),
    (lambda c: _circulant(c, 4000, 8), 296, True), (lambda c: _circulant(c, 4000, 8), 297, False),
    (lambda c: _circulant(c, 4000, 6), 296, False)])
def test_default_swendsen_wang_kernel(fake, make, R, hooks):
    """The hooking kernel runs where it is the faster one, which depends on the
    bonds, the replicas an SM and the order of the sites."""
    g = make(fake.ctx)
    fake.fake_reset()
    N.sw_run(g, np.ones((R, g.n), np.int8), [1.0], [1], seed=1)
    assert (b"sw_hook_kernel" in fake.fake_launches()) == hooks


@pytest.mark.parametrize("make,R,shape", [
    (lambda c: _lattice(c, 33), 100, (1, 288)), (lambda c: _lattice(c, 47), 100, (1, 576)),
    (lambda c: _lattice(c, 128), 100, (16, 256)),
    (lambda c: _lattice(c, 128), 256, (10, 512)), (lambda c: _lattice(c, 128), 400, (9, 512)),
    (lambda c: _lattice(c, 128), 512, (6, 512)), (lambda c: _lattice(c, 128), 832, (5, 512)),
    (lambda c: _lattice(c, 64), 256, (16, 256)), (lambda c: _circulant(c, 10000, 8), 400, (11, 512)),
    (lambda c: _circulant(c, 4000, 4), 100, (15, 512)),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(10000, 3, seed=4)[0])), 100, (16, 512)),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(2600, 3, seed=4)[0])), 100, (10, 256))])
def test_default_shape_of_the_bitpacked_kernel(fake, make, R, shape):
    """Threads follow the largest class of a part, which on graphs without
    locality is several times its share."""
    g = make(fake.ctx)
    st = N.sa_run(g, np.ones((R, g.n), np.int8), [1.0], [1], seed=1, kernel="bitpacked")
    assert (st["cluster"], st["threads"]) == shape


@pytest.mark.parametrize("make,T,R,threads", [
    (lambda c: _lattice(c, 16), 16, 64, 512), (lambda c: _lattice(c, 16), 32, 1024, 256),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(900, 3, seed=4)[0])), 16, 20, 256),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(1200, 3, seed=4)[0])), 16, 20, 512)])
def test_default_threads_of_the_slice_split_kernel(fake, make, T, R, threads):
    g = make(fake.ctx)
    st = N.sqa_run(g, np.ones((R, T, g.n), np.int8), 1.0, [1.0], [0.5], [1], seed=1, kernel="bitpacked")
    assert (st["cluster"], st["threads"]) == (1, threads)


@pytest.mark.parametrize("make,T,R", [
    (lambda c: _lattice(c, 8), 0, 64), (lambda c: _lattice(c, 33), 0, 100), (lambda c: _lattice(c, 128), 0, 400),
    (lambda c: _lattice(c, 32), 0, 256),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(4096, 3, seed=4)[0])), 16, 8),
    (lambda c: _lattice(c, 16), 16, 64)])
def test_the_tuner_times_the_default_shape(fake, make, T, R):
    """On the stand-in every candidate takes the same time, so a tuned call keeps
    the untuned one's shape, if that was a candidate at all."""
    shapes = []
    for tune in (False, True):
        g = make(fake.ctx)
        if T:
            st = N.sqa_run(g, np.ones((R, T, g.n), np.int8), 1.0, [1.0], [0.5], [4], seed=1, kernel="bitpacked", tune=tune)
        else:
            st = N.sa_run(g, np.ones((R, g.n), np.int8), [1.0], [4], seed=1, kernel="bitpacked", tune=tune)
        assert st["tuned"] == tune
        shapes.append((st["cluster"], st["threads"]))
    assert shapes[0] == shapes[1]


@pytest.mark.parametrize("make,T,groups,cluster", [
    (lambda c: _lattice(c, 32), 4, 8, 1), (lambda c: _lattice(c, 36), 4, 8, 5), (lambda c: _lattice(c, 36), 32, 74, 1),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(4096, 3, seed=4)[0])), 4, 7, 16),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(4096, 3, seed=4)[0])), 4, 8, 10),
    (lambda c: N.Graph(c, *I.augmented_csr(I.random_regular_pm_j(4096, 3, seed=4)[0])), 32, 128, 1),
    (lambda c: _circulant(c, 4000, 6), 32, 22, 6)])
def test_default_cluster_of_the_slice_split_kernel(fake, make, T, groups, cluster):
    """A cluster size with which all groups run at once, where that beats one CTA
    a group."""
    g = make(fake.ctx)
    R = groups * {4: 16, 32: 2}[T]
    st = N.sqa_run(g, np.ones((R, T, g.n), np.int8), 1.0, [1.0], [0.5], [1], seed=1, kernel="bitpacked")
    assert st["cluster"] == cluster


def test_a_partition_that_does_not_fit_is_tried_once(fake):
    """Later calls go straight to the cluster that fits: host work between a
    call's events would count as its time."""
    g = _circulant(fake.ctx, 40000, 8)
    s = np.ones((400, g.n), np.int8)
    N.sa_run(g, s, [1.0], [1], seed=1, kernel="bitpacked")
    fake.fake_fail_new(0, 64 * 1024)  # a plan's tables are larger
    N.sa_run(g, s, [1.0], [1], seed=1, kernel="bitpacked", first_sweep=1)
    pending = fake.fake_new_pending()
    fake.fake_fail_new(-1, 0)
    assert pending
