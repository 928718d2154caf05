"""CPU tests of what the host code asks of the device: the library's object files
linked against a CUDA runtime that only keeps a log (host_checks/fake_cudart.cpp).
No kernel runs, so these cover sizes, launches and call order alone."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def bind(so):
    from asmooth_gb300 import _lib

    lib = C.CDLL(so)
    for name, (res, args) in _lib.SIGNATURES.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.fake_log.restype = C.c_char_p
    lib.fake_counts.argtypes = [C.c_uint32] + 3 * [C.c_ulonglong]
    lib.fake_largest.argtypes = [C.c_size_t]
    lib.path = so
    return lib


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from asmooth_gb300 import build as B

    objs = [os.path.join(B.CSRC, "_build", u + ".o") for u in B.UNITS]
    B.build(force=not all(os.path.exists(o) and os.path.getmtime(o) >= B._sources_mtime() for o in objs))
    so = str(tmp_path_factory.mktemp("fake") / "libasg_fake.so")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc())))
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", B.CSRC, "-I",
                    os.path.join(cuda, "include"), os.path.join(HERE, "host_checks", "fake_cudart.cpp"),
                    *objs, "-o", so, "-lpthread"], check=True, capture_output=True)
    return bind(so)


@pytest.fixture
def fresh_fake(fake, tmp_path):
    """the library as in a process that has made no call yet"""
    return bind(shutil.copy(fake.path, str(tmp_path / "libasg_fresh.so")))


@pytest.fixture(autouse=True)
def fresh(fake):
    fake.fake_counts(0, 0, 0, 0)
    fake.fake_fastest(10 ** 6)
    fake.fake_spin(0)
    fake.fake_largest(2 ** 64 - 1)
    fake.fake_clear()


def log(fake):
    lines = [ln.split() for ln in fake.fake_log().decode().splitlines()]
    fake.fake_clear()
    return lines


def context(fake):
    h = C.c_void_p()
    assert fake.asg_create(C.byref(h), 0) == 0
    return h


def batch(fake, ctx, sizes, ncs=(8,)):
    """a batch of cubes of these particle counts, positions all zero"""
    k = len(sizes)
    n = np.asarray(sizes, np.int32)
    lo, hi = np.zeros(k, np.float32), np.full(k, 10, np.float32)
    nc = np.asarray(ncs, np.int32)
    b = C.c_void_p()
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    assert fake.asg_batch_create(ctx, k, p(n), None, p(lo), p(hi), p(hi), p(nc), len(nc), -1, C.byref(b)) == 0
    return b


def boxes_short(lines):
    return [ln for ln in lines if ln[0] == "boxes" and int(ln[1]) > int(ln[2])]


@pytest.mark.parametrize("leaf", ["", "1", "17", "24", "32"])
def test_tuned_leaf_sizes_fit_the_box_array(fake, monkeypatch, leaf):
    """The tuner's index builds keep to the tree's box array whatever leaf size the
    context starts from, and so does a later, larger batch of the same context, which
    starts from the leaf size that the first one chose (the largest here)."""
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    ctx = context(fake)
    for sizes in ([3000, 2000], [90000, 4000], [200000]):
        b = batch(fake, ctx, sizes)
        chosen = C.c_int(0)
        assert fake.asg_batch_tune(b, C.byref(chosen), None) == 0 and chosen.value == 32
        assert fake.asg_batch_run(b) == 0
        fake.asg_batch_destroy(b)
    lines = log(fake)
    assert sum(ln[0] == "boxes" for ln in lines) > 100
    assert not boxes_short(lines)
    fake.asg_destroy(ctx)


@pytest.mark.parametrize("pairs,tiles", [
    ((10 ** 6, 10 ** 6, 10 ** 6), "own"),
    ((8 * 2 ** 20, 2 ** 22, 2 ** 21), "own"),  # the line of deposit_wide_pairs for few particles
    ((8 * 2 ** 20 + 1, 2 ** 22, 2 ** 21), "wide"),
    ((2 ** 31, 2 ** 30, 2 ** 29), "wide"),
    ((2 ** 33, 2 ** 31 - 1, 2 ** 30), "wide"),
    ((2 ** 33, 2 ** 31, 2 ** 31 - 1), "large")])
def test_captured_deposit_takes_the_planned_tiles(fake, pairs, tiles):
    """A batch item with many pairs, or with more than 32 bits number, takes larger
    tiles in the planning pass, and so it does in the graph, whose capture allocates
    nothing."""
    ctx = context(fake)
    b = batch(fake, ctx, [5000, 4000], ncs=(16, 32))
    fake.fake_counts(1000, *pairs)
    assert fake.asg_batch_run(b) == 0
    lines = log(fake)
    at = [ln[0] for ln in lines].index("capture")
    want = {"own": "k_deposit_mmaILi6ELb0E", "wide": "k_deposit_mmaILi6ELb1E", "large": "k_deposit_items"}[tiles]
    for part in (lines[:at], lines[at:]):
        ran = [ln[1] for ln in part if ln[0] == "launch" and "k_deposit_" in ln[1]]
        assert len(ran) == 2 and all(want in k for k in ran)
    assert not any(ln[0] == "malloc" for ln in lines[at:])
    fake.asg_batch_destroy(b)
    fake.asg_destroy(ctx)


def test_tuned_context_walks_the_tree_it_built(fake):
    """The tuner leaves the largest item loaded, with a tree of the last leaf size it
    timed; calls on that set walk that tree, whatever leaf size was chosen."""
    ctx = context(fake)
    b = batch(fake, ctx, [3000, 2000])
    fake.fake_fastest(2)
    chosen, groups = C.c_int(0), C.c_int(0)
    assert fake.asg_batch_tune(b, C.byref(chosen), None) == 0 and chosen.value == 16
    assert fake.asg_run_fof(ctx, 0.5, C.byref(groups)) == 0
    halo = np.zeros(5, np.float32)
    assert fake.asg_run_mark_halos(ctx, halo.ctypes.data, 1, None, None) == 0
    assert fake.asg_get_knn(ctx, None, None) == 0
    trees = [ln for ln in log(fake) if ln[0] == "tree"]
    assert ["k_mark_halos" in trees[-2][1], "k_knn_ties" in trees[-1][1]] == [True, True]
    built = [int(t[2]) for t in trees if "k_gather" in t[1]][-1]
    assert [int(t[2]) for t in trees[-3:]] == 3 * [built]
    fake.asg_batch_destroy(b)
    fake.asg_destroy(ctx)


def test_tuner_that_fails_leaves_the_configuration(fake, monkeypatch):
    """... and no graph that holds buffers which it may have moved."""
    monkeypatch.setenv("ASG_LEAF_SIZE", "24")
    ctx = context(fake)
    b = batch(fake, ctx, [3000])
    v = [C.c_int(0) for _ in range(8)]
    assert fake.asg_batch_config(b, *[C.byref(t) for t in v[:4]]) == 0 and v[0].value == 24
    assert fake.asg_batch_run(b) == 0
    fake.fake_counts(10, 2 ** 33, 2 ** 33, 2 ** 33)  # more pairs than any tile shape can number
    assert fake.asg_batch_tune(b, None, None) != 0
    assert fake.asg_batch_config(b, *[C.byref(t) for t in v[4:]]) == 0
    assert [t.value for t in v[4:]] == [t.value for t in v[:4]]
    fake.fake_counts(10, 100, 100, 100)
    log(fake)
    assert fake.asg_batch_run(b) == 0
    assert ["capture"] in log(fake)
    fake.asg_batch_destroy(b)
    fake.asg_destroy(ctx)


@pytest.mark.parametrize("density_only", [0, 1])
def test_small_deposits_take_little_memory(fake, density_only):
    """A deposit's partial tiles are sized by its pairs: a few MB for a few particles."""
    ctx = context(fake)
    x = np.zeros((100, 3), np.float32)
    assert fake.asg_load_particles_device(ctx, x.ctypes.data, None, None, None, 100, 0.0, 1.0) == 0
    fake.fake_counts(50, 1000, 500, 300)
    log(fake)
    nc = np.asarray([16], np.int32)
    assert fake.asg_run_deposit(ctx, 1.0, nc.ctypes.data, 1, -1, 0, None, density_only, None) == 0
    assert sum(int(ln[1]) for ln in log(fake) if ln[0] == "malloc") < 4 << 20
    fake.asg_destroy(ctx)


@pytest.mark.parametrize("n_alone", [False, True])
def test_items_fit_the_room_for_them(fake, n_alone):
    """deposit_max_items covers the items that k_tile_items makes of any split of the
    pairs over the tiles, also when a plan has room for more pairs than there are."""
    room = getattr(fake, "_ZN3asg17deposit_max_itemsEijib")
    room.restype, room.argtypes = C.c_uint32, [C.c_int, C.c_uint32, C.c_int, C.c_bool]
    share = 4 * 24 * 152 // (2 if n_alone else 1)
    rng = np.random.default_rng(2)
    for pairs in [0, 1, 63, 64, 65, 10_000, 500_000, 933_888, 933_889, 20_000_000, 2 ** 31 - 1]:
        for most in (2048, 4096, 8192):
            seg = min((pairs // share + 64) & ~63, most)
            for tiles in (1, 7, 3000):
                even = np.full(tiles, pairs // tiles)
                even[0] += pairs - even.sum()
                some = rng.multinomial(pairs, rng.dirichlet(np.full(tiles, 0.1)))
                # as many tiles as there can be with one pair over a full item
                full = np.zeros(tiles, np.int64)
                k = min(tiles, pairs // (seg + 1))
                full[:k] = seg + 1
                full[0] += pairs - full.sum()
                for c in (even, some, full):
                    items = int(np.maximum(1, -(-c // seg)).sum())
                    for planned in (pairs, min(pairs + pairs // 16 + 4096, 2 ** 32 - 1)):
                        assert items <= room(tiles, planned, most, n_alone)


def test_headroom_stays_within_the_sort(fake):
    """A batch's plan has room for a sixteenth more entries, but no more than the sort
    can number (a larger count would be negative there, and nothing sorted)."""
    room = getattr(fake, "_ZN3asg16deposit_headroomEj")
    room.restype, room.argtypes = C.c_uint32, [C.c_uint32]
    for n in [0, 1, 1000, 10 ** 9, 2_021_157_000, 2_021_157_300, 2 ** 31 - 5000, 2 ** 31 - 1]:
        assert room(n) == min(n + n // 16 + 4096, 2 ** 31 - 1) >= n


def test_tuner_times_no_setting_twice(fake):
    """Leaves of 16 run the search in blocks of their own, so the warps per block are
    no setting there: 3 x 2 settings with leaves of 16, 3 x 2 x 2 with each other size,
    two passes each."""
    ctx = context(fake)
    b = batch(fake, ctx, [3000])
    assert fake.asg_batch_tune(b, None, None) == 0
    searches = [tuple(ln[1:4]) for ln in log(fake) if ln[0] == "launch" and "k_knn_t33" in ln[1]]
    assert len(searches) == 2 * (6 + 12 + 12)
    fake.asg_batch_destroy(b)
    fake.asg_destroy(ctx)


def test_every_persistent_kernel_gets_its_attributes(fresh_fake):
    """The deposit kernels share a signature; each has its shared memory and carve-out
    set before its first launch."""
    ctx = context(fresh_fake)
    x = np.zeros((100, 3), np.float32)
    assert fresh_fake.asg_load_particles_device(ctx, x.ctypes.data, None, None, None, 100, 0.0, 1.0) == 0
    nc = np.asarray([16], np.int32)
    for density_only, pairs in ((0, 1000), (1, 1000), (0, 2 ** 30), (0, 2 ** 33)):
        fresh_fake.fake_counts(50, pairs, pairs, pairs // 8)
        assert fresh_fake.asg_run_deposit(ctx, 1.0, nc.ctypes.data, 1, -1, 0, None, density_only, None) == 0
    lines = log(fresh_fake)
    kernels = {ln[1] for ln in lines if ln[0] == "launch" and "k_deposit_" in ln[1]}
    assert len(kernels) == 4
    smem, carveout = "8", "9"  # cudaFuncAttribute
    for k in kernels:
        first = next(i for i, ln in enumerate(lines) if ln[:2] == ["launch", k])
        assert {ln[2] for ln in lines[:first] if ln[:2] == ["attr", k]} == {smem, carveout}
    fresh_fake.asg_destroy(ctx)


def test_preparing_call_loads_what_a_search_launches(fresh_fake):
    """asg_neighbor_search_noalloc: the preparing call loads the kernels of every
    particle count (a first load later may take device memory), allocates nothing, and
    the fixed scratch holds every count."""
    fake = fresh_fake
    assert fake.asg_neighbor_search_noalloc(None, 0, 0.0, 0.0, None, None, None) == 0
    loaded = {ln[1] for ln in log(fake) if ln[0] == "load"}
    a = np.zeros(3 * 32768, np.float32)
    p = C.c_void_p(a.ctypes.data)
    edges = [33, 64, 1024, 4099, 4864, 4865, 8192, 8193, 16384, 16385, 20000, 24320, 24321, 32767, 32768]
    for n in edges + list(range(33, 32768, 487)):
        assert fake.asg_neighbor_search_noalloc(p, n, 0.0, 1.0, p, p, None) == 0
    lines = log(fake)
    launched = {ln[1] for ln in lines if ln[0] == "launch"}
    assert len(launched) > 10 and launched <= loaded
    assert not any(ln[0] == "malloc" for ln in lines)


def test_times_are_read_from_events_that_are_done(fake):
    """A call that polls for its results returns when a kernel has stored them, which
    says nothing of the events recorded before it: times are read after a wait for them,
    and an event that is not done would leave an error for the next call."""
    fake.fake_spin(1)
    ctx = context(fake)
    assert fake.asg_set_timing(ctx, 1) == 0
    x = np.zeros((100, 3), np.float32)
    ms = np.zeros(10)
    for _ in range(2):
        assert fake.asg_load_particles_device(ctx, x.ctypes.data, None, None, None, 100, 0.0, 1.0) == 0
        assert fake.asg_run_neighbor_search(ctx) == 0
    assert fake.asg_phase_ms(ctx, ms.ctypes.data) == 0
    assert (ms[[0, 1, 2, 4]] > 0).all()  # index, search, ties, density
    b = batch(fake, ctx, [3000])
    graph_ms = C.c_double(0.0)
    assert fake.asg_batch_run(b) == 0 and fake.asg_batch_run(b) == 0
    assert fake.asg_batch_stats(b, C.byref(graph_ms), None, None) == 0 and graph_ms.value > 0
    fake.asg_batch_destroy(b)
    fake.asg_destroy(ctx)


def test_out_of_memory_leaves_nothing_half_loaded(fake):
    """A load that finds no memory takes the loaded set's arrays with it, a decode the
    decoded particles', a deposit the mesh's: calls on them are refused, and no kernel
    runs on arrays that are gone."""
    STATE, NOMEM, ARG = -10, -3, -1
    ctx = context(fake)
    x = np.zeros((200_000, 3), np.float32)
    p, out = x.ctypes.data, np.zeros(200_000, np.float32).ctypes.data
    n_out, groups = C.c_int(0), C.c_int(0)
    nc = np.asarray([16], np.int32)

    def load(n):
        return fake.asg_load_particles_device(ctx, p, None, None, None, n, 0.0, 1.0)

    def deposit():
        return fake.asg_run_deposit(ctx, 1.0, nc.ctypes.data, 1, -1, 0, None, 0, None)

    assert load(100) == 0 and fake.asg_run_neighbor_search(ctx) == 0 and deposit() == 0
    assert fake.asg_load_periodic_cube_device(ctx, p, None, 100, 1.0, 0.1, None, None) != NOMEM
    assert load(100) == 0 and fake.asg_run_neighbor_search(ctx) == 0
    for largest in (1 << 20, 5 << 20):  # no array of the larger set fits; some do
        fake.fake_largest(largest)
        assert load(200_000) == NOMEM
        log(fake)
        assert fake.asg_run_neighbor_search(ctx) == STATE and deposit() == STATE
        assert fake.asg_get_knn(ctx, None, None) == STATE
        assert fake.asg_run_fof(ctx, 0.5, C.byref(groups)) == STATE
        assert fake.asg_store_fields_device(ctx, out, out, None) == STATE
        assert not [ln for ln in log(fake) if ln[0] == "launch"]
    assert fake.asg_load_periodic_cube_device(ctx, p, None, 200_000, 1.0, 0.1, None, None) == NOMEM
    log(fake)
    assert fake.asg_load_decoded_periodic(ctx, 1.0, 0.1, C.byref(n_out), None) == STATE
    assert fake.asg_copy_decoded(ctx, p) == STATE
    assert not [ln for ln in log(fake) if ln[0] == "launch"]
    assert load(100) == 0
    nc[0] = 200
    assert deposit() == NOMEM
    log(fake)
    assert fake.asg_run_normalise(ctx, 0) == ARG
    assert fake.asg_copy_mesh(ctx, 0, out) == ARG
    assert not [ln for ln in log(fake) if ln[0] == "launch"]
    fake.fake_largest(2 ** 64 - 1)
    assert load(200_000) == 0 and fake.asg_run_neighbor_search(ctx) == 0
    fake.asg_destroy(ctx)
