"""The library's host code on paths a GPU run cannot be brought to: allocations
that fail, a second device, clusters that do not fit, options that are refused.
Its objects are linked with fake_cudart.cpp, a runtime whose device memory is
host memory and whose kernels do nothing, and driven through the C ABI."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import vespa_b200 as vb
from vespa_b200 import _lib
from vespa_b200 import problem as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vespa.jl_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    # the library's objects, built with it (a no-op where they are up to date)
    subprocess.run(["make", "-C", CSRC, f"-j{os.cpu_count()}", "all"], check=True, capture_output=True)
    so = str(tmp_path_factory.mktemp("fake") / "libvespa_fake.so")
    objs = [os.path.join(CSRC, "_build", f) for f in os.listdir(os.path.join(CSRC, "_build"))
            if f.endswith(".o")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-o", so,
                    "-I", os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "fake_cudart.cpp"),
                    *objs, "-lpthread"], check=True, capture_output=True)
    L = C.CDLL(so)
    for name, args in _lib.SIGNATURES.items():
        getattr(L, name).argtypes = args
    for f in ("fake_device_live", "fake_pinned_live", "fake_plain_bytes", "fake_refused", "fake_launched"):
        getattr(L, f).restype = C.c_longlong
    L.fake_launched.argtypes = [C.c_char_p]
    L.fake_refused.argtypes = [C.c_char_p, C.c_size_t]
    L.fake_fail_device_alloc.argtypes = L.fake_fail_graph_launch.argtypes = [C.c_longlong]
    L.fake_host_alloc.restype = C.c_void_p
    L.fake_host_alloc.argtypes = [C.c_size_t]
    L.fake_host_free.argtypes = [C.c_void_p]
    L.vb_last_error.argtypes = [C.c_char_p, C.c_size_t]
    return L


@pytest.fixture
def ctx(fake):
    fake.fake_reset()
    c = C.c_void_p()
    assert fake.vb_ctx_create(0, C.byref(c)) == 0
    yield c
    fake.fake_reset()
    fake.vb_ctx_destroy(c)


def error(L):
    buf = C.create_string_buffer(512)
    L.vb_last_error(buf, 512)
    return buf.value.decode()


def make_grid(L, ctx, dims, precision=_lib.FP64, bc=P.Periodic):
    prob = P.smooth_random_problem(dims, seed=1)
    prob.bcs = tuple((bc, bc) for _ in dims)
    g = C.c_void_p()
    rc = L.vb_grid_create(ctx, C.byref(vb.simulation.problem_desc(prob)), precision, C.byref(g))
    assert rc == 0, error(L)
    return g


def test_adjoint_scratch_matches_the_kernels_that_use_it(fake, ctx):
    """Only 2D grids whose stage keeps its face adjoints on chip go without the
    three scratch arrays; longer or thinner ones take the kernels that write
    them."""
    live = []
    for dims, on_chip in (((64, 4), True), ((4, 4000), True), ((4, 65536), False), ((65536, 1), False),
                          ((8, 65536), True), ((1, 2 ** 24 + 1), False)):
        g = make_grid(fake, ctx, dims)
        before = fake.fake_device_live()
        a = C.c_void_p()
        assert fake.vb_adjoint_create(g, 4, 2, C.byref(a)) == 0, error(fake)
        live.append(fake.fake_device_live() - before)
        assert live[-1] == live[0] + (0 if on_chip else 3), dims
        if max(dims) < 2 ** 24:
            U = np.ones((5, int(np.prod(dims))))
            fake.fake_reset()
            assert fake.vb_adjoint_step(a, 0.1, _lib.dptr(U), _lib.dptr(U)) == 0, error(fake)
            assert (fake.fake_launched(b"k_adj_plane") > 0) == on_chip
            assert (fake.fake_launched(b"k_adj_face") > 0) == (not on_chip)
        fake.vb_adjoint_destroy(a)
        assert fake.fake_device_live() == before
        fake.vb_grid_destroy(g)


def faces(nf):
    r = np.random.default_rng(nf)
    return r.random((nf, 5)) + 0.5, r.random((nf, 5)) + 0.5, r.integers(1, 4, nf).astype(np.int32), np.zeros((nf, 5))


def hllc(L, ctx, WL, WR, axis, F):
    return L.vb_hllc_faces(ctx, len(axis), _lib.dptr(WL), _lib.dptr(WR), _lib.i32ptr(axis), 1.4, _lib.dptr(F))


def test_copies_and_batches_go_plainly_when_no_lanes_can_be_made(fake, ctx):
    g = make_grid(fake, ctx, (64, 64, 128))
    U = np.random.default_rng(0).random((5, 64 * 64 * 128))
    back = np.zeros_like(U)
    WL, WR, axis, F = faces(40000)
    pinned = fake.fake_pinned_live()
    for i in range(32):  # 40 MB of copies and 5 MB of faces a round: beyond every threshold
        fake.fake_fail_pinned(i < 16)  # first no page-locked memory, then none on the device
        fake.fake_fail_device(i >= 16)
        assert fake.vb_grid_upload(g, _lib.dptr(U)) == 0, error(fake)
        assert fake.vb_grid_download(g, _lib.dptr(back)) == 0, error(fake)
        assert np.array_equal(U, back)
        assert hllc(fake, ctx, WL, WR, axis, F) == 0, error(fake)
        assert fake.fake_pinned_live() == pinned  # nothing half made is kept
        U += 1.0
    fake.fake_fail_device(0)
    fake.vb_grid_destroy(g)


def test_pinned_and_overlapping_face_batches_stay_whole(fake, ctx):
    """One launch for the batch; the lanes would take one per 8192 faces."""
    nf = 40000

    def launches(WL, WR, axis, F):
        before = fake.fake_launched(b"k_hllc_faces")
        assert hllc(fake, ctx, WL, WR, axis, F) == 0, error(fake)
        return fake.fake_launched(b"k_hllc_faces") - before

    WL, WR, axis, F = faces(nf)
    for _ in range(64):  # by then pageable batches are staged
        staged = launches(WL, WR, axis, F)
    assert staged == -(-nf // 8192)
    for which in range(3):
        arrays = [WL, WR, F]
        p = fake.fake_host_alloc(8 * 5 * nf)
        arrays[which] = np.ctypeslib.as_array((C.c_double * (5 * nf)).from_address(p)).reshape(nf, 5)
        assert launches(arrays[0], arrays[1], axis, arrays[2]) == 1
        fake.fake_host_free(p)
    both = np.random.default_rng(1).random((nf + 10, 5))
    assert launches(both[10:], WR, axis, both[:nf]) == 1
    assert launches(WL, both[:nf], axis, both[10:]) == 1
    assert launches(WL, WR, axis, WL) == 1


def test_lanes_are_made_only_once_large_arrays_add_up(fake, ctx):
    nf = 200000  # 24.8 MB a batch
    WL, WR, axis, F = faces(nf)
    pinned = fake.fake_pinned_live()
    made = []
    for _ in range(12):
        assert hllc(fake, ctx, WL, WR, axis, F) == 0, error(fake)
        made.append(fake.fake_pinned_live() - pinned)
    assert made[:10] == [0] * 10 and made[11] == 8, made  # 256 MiB after ten batches


@pytest.mark.parametrize("dims", [(64, 48), (20, 12, 9)])
def test_a_refused_option_leaves_the_grid_as_it_was(fake, ctx, dims):
    g = make_grid(fake, ctx, dims)

    def kernels():
        fake.fake_reset()
        assert fake.vb_run_steps_async(g, 1) == 0, error(fake)
        return [fake.fake_launched(k) for k in (b"k_march", b"k_stage_plane_f64", b"k_stage_generic")]

    for chosen in ("auto", "cell"):
        assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, _lib.KERNELS[chosen]) == 0
        before = kernels()
        assert sum(before)
        for bad, code in ((_lib.KERNELS["tiled"], _lib.VB_ENOTSUP), (7, _lib.VB_EINVAL), (-1, _lib.VB_EINVAL)):
            assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, bad) == code
            assert kernels() == before, (chosen, bad)
    fake.vb_grid_destroy(g)


def test_a_second_device_gets_its_own_kernel_opt_ins(fake, ctx):
    """Shared-memory and cluster-size opt-ins belong to a device: one run on the
    first must not stand for the second."""
    fake.fake_devices(2)
    other = C.c_void_p()
    assert fake.vb_ctx_create(1, C.byref(other)) == 0
    grids = [((64, 64), _lib.FP64, "auto"), ((300,), _lib.FP64, "auto"), ((256, 64), _lib.FP64, "tiled"),
             ((512, 4096), _lib.MIXED, "auto"), ((48, 48, 48), _lib.FP64, "auto"), ((48, 48, 48), _lib.MIXED, "auto"),
             ((48, 47, 48), _lib.FP64, "auto")]
    for c in (ctx, other):
        for dims, prec, kind in grids:
            g = make_grid(fake, c, dims, prec)
            assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, _lib.KERNELS[kind]) == 0, error(fake)
            for bflux in (0, 1):
                assert fake.vb_bflux_enable(g, bflux) == 0, error(fake)
                assert fake.vb_run_steps_async(g, 2) == 0, (dims, error(fake))
            if prec == _lib.FP64 and len(dims) == 2:
                a = C.c_void_p()
                assert fake.vb_adjoint_create(g, 2, 1, C.byref(a)) == 0, error(fake)
                U = np.ones((5, int(np.prod(dims))))
                assert fake.vb_adjoint_step(a, 0.1, _lib.dptr(U), _lib.dptr(U)) == 0, error(fake)
                fake.vb_adjoint_destroy(a)
            fake.vb_grid_destroy(g)
        b = C.c_void_p()
        prob = P.smooth_random_problem((32, 32, 32), seed=1)
        assert fake.vb_batch_create(c, 1, C.byref(vb.simulation.problem_desc(prob)), _lib.FP64, C.byref(b)) == 0
        assert fake.vb_batch_run_steps_async(b, 2) == 0, error(fake)
        fake.vb_batch_destroy(b)
    why = C.create_string_buffer(256)
    assert fake.fake_refused(why, 256) == 0, why.value
    fake.vb_ctx_destroy(other)


def test_grids_march_only_where_their_cluster_fits(fake, ctx):
    for clusters, kernel in ((1, b"k_march"), (0, b"k_stage_plane_f64")):
        fake.fake_clusters(clusters)
        g = make_grid(fake, ctx, (64, 64))
        for _ in range(2):
            assert fake.vb_run_steps_async(g, 2) == 0, error(fake)
            assert fake.fake_launched(kernel) > 0
            assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, 0) == 0
        assert fake.fake_refused(None, 0) == 0
        fake.vb_grid_destroy(g)
        fake.fake_reset()


def gravity_desc(bc, precond=0, maxiter=100):
    d = _lib.GravityDesc()
    d.G, d.tol, d.maxiter, d.project_mean, d.precond, d.flags = 1.0, 1e-8, maxiter, 1, precond, 0
    for a in range(3):
        d.bc_lo[a] = d.bc_hi[a] = bc
    return d


@pytest.mark.parametrize("start", [None, (_lib.BC_OUTFLOW, 0), (_lib.BC_PERIODIC, 0)])
def test_gravity_enable_that_fails_leaves_what_was_there(fake, ctx, start):
    """Each allocation of a (re-)enable made to fail in turn: the error is
    reported, gravity that was on stays on with its settings, and the next call
    has every buffer that one without failures has."""
    wanted = C.byref(gravity_desc(_lib.BC_PERIODIC, precond=1))

    def grid():
        g = make_grid(fake, ctx, (32, 32, 32))
        if start:
            assert fake.vb_gravity_enable(g, C.byref(gravity_desc(*start))) == 0, error(fake)
        return g

    phi = np.zeros(32 ** 3)
    base = fake.fake_device_live()
    g = grid()
    assert fake.vb_gravity_enable(g, wanted) == 0, error(fake)
    full = fake.fake_device_live()
    fake.vb_grid_destroy(g)
    assert fake.fake_device_live() == base
    fails = 0
    while True:
        g = grid()
        fake.fake_fail_device_alloc(fails)
        rc = fake.vb_gravity_enable(g, wanted)
        fake.fake_fail_device_alloc(-1)
        if rc == 0:
            fake.vb_grid_destroy(g)
            break
        assert rc == _lib.VB_ENOMEM, error(fake)
        cube = start and start[0] == _lib.BC_PERIODIC
        fake.fake_reset()
        if start:  # still on, still as it was set up
            assert fake.vb_gravity_phi(g, _lib.dptr(phi)) == 0, error(fake)
            assert fake.vb_gravity_set_phi(g, _lib.dptr(phi)) == 0, error(fake)
            assert (fake.fake_launched(b"k_cube_accel") > 0) == bool(cube), fails
        else:
            assert fake.vb_gravity_phi(g, _lib.dptr(phi)) == _lib.VB_EINVAL
        assert fake.vb_gravity_enable(g, wanted) == 0, error(fake)
        assert fake.fake_device_live() == full, fails
        fake.vb_grid_destroy(g)
        assert fake.fake_device_live() == base
        fails += 1
    assert fails >= 4


CELL, TILED, PLANE, MARCH = 1, 2, 3, 4


def kernel_of(L, g):
    v = C.c_int64()
    assert L.vb_grid_get_option(g, _lib.OPT_KERNEL, C.byref(v)) == 0
    return v.value


def test_the_reported_kernel_is_the_one_that_runs(fake, ctx):
    """VB_OPT_KERNEL against the launches of a step, as boundary fluxes and
    gravity come and go."""
    names = {CELL: b"k_stage_generic", TILED: b"k_stage_tiled", PLANE: b"k_stage_plane", MARCH: b"k_march"}

    def check(g, want):
        assert kernel_of(fake, g) == want
        fake.fake_reset()
        assert fake.vb_run_steps_async(g, 1) == 0, error(fake)
        ran = {k for k, n in names.items() if fake.fake_launched(n)}
        assert ran == {want}

    # (dims, precision, selector): plain, with outer fluxes, with interior ones, with gravity
    for dims, prec, sel, kernels in [
            ((64, 48), _lib.FP64, 0, (MARCH, CELL, CELL, CELL)),
            ((64, 48), _lib.FP64, CELL, (CELL, CELL, CELL, CELL)),
            ((300, 301), _lib.FP64, 0, (PLANE, CELL, CELL, CELL)),
            ((512, 1184), _lib.FP64, 0, (PLANE, TILED, CELL, CELL)),
            ((512, 1176), _lib.FP64, 0, (PLANE, CELL, CELL, CELL)),
            ((256, 64), _lib.FP64, TILED, (TILED, TILED, CELL, CELL)),
            ((512, 1200), _lib.MIXED, 0, (TILED, TILED, CELL, CELL)),
            ((48, 47, 48), _lib.FP64, 0, (TILED, TILED, CELL, TILED)),
            ((48, 47, 48), _lib.MIXED, 0, (TILED, TILED, CELL, TILED)),
            ((20, 12, 9), _lib.FP64, 0, (CELL, CELL, CELL, CELL))]:
        g = make_grid(fake, ctx, dims, prec)
        assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, sel) == 0, error(fake)
        for mode, want in zip((_lib.BFLUX_OFF, _lib.BFLUX_OUTER, _lib.BFLUX_INTERIOR), kernels):
            assert fake.vb_bflux_enable(g, mode) == 0, error(fake)
            check(g, want)
        assert fake.vb_bflux_enable(g, _lib.BFLUX_OFF) == 0
        assert fake.vb_gravity_enable(g, C.byref(gravity_desc(_lib.BC_OUTFLOW, maxiter=0))) == 0, error(fake)
        assert kernel_of(fake, g) == kernels[3]
        fake.vb_grid_destroy(g)


@pytest.mark.parametrize("dims,kind,prec", [((512, 1184), "auto", _lib.FP64), ((64, 48), "auto", _lib.FP64),
                                            ((256, 64), "tiled", _lib.FP64), ((48, 47, 48), "auto", _lib.MIXED)])
def test_autotune_times_only_grids_whose_steps_are_tiled(fake, ctx, dims, kind, prec):
    g = make_grid(fake, ctx, dims, prec)
    assert fake.vb_grid_set_option(g, _lib.OPT_KERNEL, _lib.KERNELS[kind]) == 0
    kz, best, ms = C.c_int64(), C.c_int64(), C.c_double(7.0)
    assert fake.vb_grid_get_option(g, _lib.OPT_TILE_KZ, C.byref(kz)) == 0
    tiled = kernel_of(fake, g) == TILED
    fake.fake_reset()
    assert fake.vb_grid_autotune(g, 2, C.byref(best), C.byref(ms)) == 0, error(fake)
    if tiled:
        assert fake.fake_launched(b"k_stage_tiled") > 0 and ms.value > 0.0
    else:
        assert fake.fake_launched(b"k_") == 0 and ms.value == 0.0 and best.value == kz.value
    fake.vb_grid_destroy(g)
    g = make_grid(fake, ctx, dims, prec)  # and nothing is kept for later grids of its kind
    kept = C.c_int64()
    assert fake.vb_grid_get_option(g, _lib.OPT_TILE_KZ, C.byref(kept)) == 0
    assert kept.value == best.value
    fake.vb_grid_destroy(g)


@pytest.mark.parametrize("dims,precision,kernel", [
    ((17, 17, 512), _lib.FP64, CELL), ((18, 18, 512), _lib.MIXED, CELL),  # tiles would solve 3.5, 3.2 times the cells
    ((20, 20, 512), _lib.FP64, CELL), ((20, 20, 512), _lib.MIXED, TILED),  # 2.6
    ((33, 33, 100), _lib.FP64, TILED), ((16, 16, 512), _lib.FP64, TILED), ((16, 17, 512), _lib.FP64, TILED),
    ((33, 47, 31), _lib.FP64, TILED), ((32, 32, 32), _lib.FP64, CELL)])
def test_thin_boxes_keep_the_cell_kernel(fake, ctx, dims, precision, kernel):
    g = make_grid(fake, ctx, dims, precision)
    assert kernel_of(fake, g) == kernel
    fake.vb_grid_destroy(g)


def test_long_cube_solves_come_back_to_the_host(fake, ctx):
    """Iterations beyond 512 are queued a run at a time: the third run's failure
    to start ends the solve (one run for the whole limit would not see it)."""
    for maxiter, rc in ((512, 0), (10 ** 9, _lib.VB_ECUDA)):
        g = make_grid(fake, ctx, (32, 32, 32))
        assert fake.vb_gravity_enable(g, C.byref(gravity_desc(_lib.BC_PERIODIC, 1, maxiter))) == 0, error(fake)
        fake.fake_fail_graph_launch(2)
        assert fake.vb_gravity_solve(g, None, None) == rc
        fake.fake_reset()
        fake.vb_grid_destroy(g)


def test_gravity_allocates_what_its_passes_use(fake, ctx):
    """A cube forms its right-hand side on the fly, and levels that one block
    runs in shared memory have no second array; walls bring the array back."""
    g = make_grid(fake, ctx, (32, 32, 32))
    base = fake.fake_device_live()
    assert fake.vb_gravity_enable(g, C.byref(gravity_desc(_lib.BC_PERIODIC, precond=1))) == 0, error(fake)
    # phi r p Ap field partials control; block partials, second direction, z z2;
    # two arrays a level (32, 16, 8, 4), a third on the first
    assert fake.fake_device_live() - base == 7 + 4 + 2 * 4 + 1
    assert fake.vb_gravity_enable(g, C.byref(gravity_desc(_lib.BC_OUTFLOW))) == 0, error(fake)
    assert fake.fake_device_live() - base == 7 + 4 + 2 * 4 + 1 + 1
    fake.vb_grid_destroy(g)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
def test_the_starting_chunk_fits_the_grid(fake, ctx, precision):
    """The chunk that a grid starts with can be set on a grid of its kind."""
    for dims in [(512, 512, 4), (640, 512, 3), (768, 768, 2), (512, 512, 7), (256, 256, 8), (48, 48, 48), (16, 16, 300),
                 (2048, 2), (4096, 5), (2048, 300), (512, 9)]:
        g = make_grid(fake, ctx, dims, precision)
        kz = C.c_int64()
        assert fake.vb_grid_get_option(g, _lib.OPT_TILE_KZ, C.byref(kz)) == 0
        assert kz.value <= dims[-1], (dims, kz.value)
        if kernel_of(fake, g) == TILED:
            assert fake.vb_grid_set_option(g, _lib.OPT_TILE_KZ, kz.value) == 0, (dims, error(fake))
        fake.vb_grid_destroy(g)
