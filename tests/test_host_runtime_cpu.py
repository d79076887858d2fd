"""The host runtime's bookkeeping without a GPU: the library's own objects on a
CUDA runtime for the CPU (tests/cpp/fake_cuda.cpp). Kernels do nothing there;
what is checked is that every buffer a copy or a launch names is allocated and
long enough, and when the library allocates, waits and orders its streams."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ALPHA, BETA = 0.97, 1.9


@pytest.fixture(scope="module")
def fake_library():
    r = subprocess.run(["make", "-C", os.path.join(ROOT, "tests", "cpp"), "fake"], stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout[-3000:]
    return os.path.join(ROOT, "tests", "cpp", "_bin", "libtdlb_fake_cuda.so")


@pytest.fixture
def fake(fake_library, monkeypatch):
    """The package on the CPU runtime; fake.lib has its fake_* functions."""
    import tdlbcpp_b200 as tb
    monkeypatch.setattr(tb, "_lib", None)
    monkeypatch.setattr(tb, "library_path", lambda: fake_library)
    lib = tb.load_library()
    for name in ("mallocs", "waits"):
        getattr(lib, "fake_" + name).restype = ctypes.c_longlong
    lib.fake_faults.restype = ctypes.c_char_p
    lib.fake_fail.argtypes = [ctypes.c_longlong]
    lib.fake_foreign.argtypes, lib.fake_foreign.restype = [ctypes.c_void_p], ctypes.c_longlong
    lib.fake_launches.argtypes, lib.fake_launches.restype = [ctypes.c_char_p], ctypes.c_longlong
    lib.fake_unordered.argtypes = [ctypes.c_char_p, ctypes.c_void_p, ctypes.c_longlong]
    lib.fake_unordered.restype = ctypes.c_longlong
    lib.fake_pin.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.fake_reset()
    yield tb
    lib.fake_reset()


def faults(tb):
    return tb.load_library().fake_faults().decode()


def markers(tb, n, dims, seed=1):
    rng = np.random.default_rng(seed)
    m = np.zeros(n, tb.MARKER_DTYPE)
    for name, hi in zip("ijk", dims):
        m[name] = rng.integers(0, hi, n)
    return m


def test_lists_of_changing_length_stay_in_their_buffers(fake):
    dims = (20, 24, 18)
    cu = fake.ComputeUnit(x=dims[0], y=dims[1], z=dims[2], nu=1e-3)
    cu.initialise(1.0)
    for n in (500, 1000, 5000, 5000, 3000, 6000, 6000, 0, 2000, 7000, 7000):
        cu.forcing(markers(fake, n, dims), ALPHA, BETA)
        assert not faults(fake), f"after {n} markers"
    bad = markers(fake, 9000, dims)
    bad["i"][4000] = dims[0]
    for n in (8000, 9000, 8000, 9000):
        with pytest.raises(fake.TdlbError, match="marker 4000 at"):
            cu.set_markers(bad[:n])
        np.testing.assert_array_equal(cu.read_markers(), markers(fake, 7000, dims))
        cu.forcing(markers(fake, 7000, dims), ALPHA, BETA)
        assert not faults(fake)
    cu.doubleResolutionFullCU()
    cu.initialise(1.0)
    for n in (20000, 20000, 20000):
        cu.forcing(markers(fake, n, dims), ALPHA, BETA)
        assert not faults(fake), f"after {n} markers on the doubled lattice"
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("call", [lambda cu: cu.read_moments(), lambda cu: cu.plane_xz(3), lambda cu: cu.reduce_fp64(),
                                  lambda cu: cu.doubleResolutionFullCU()])
def test_a_failed_allocation_is_told_of_once(fake, call):
    """A call without memory for its scratch fails; the same call does not then."""
    cu = fake.ComputeUnit(x=24, y=24, z=24, nu=1e-3)
    cu.initialise(1.0)
    fake.load_library().fake_fail(1)
    with pytest.raises(fake.TdlbError):
        call(cu)
    call(cu)
    cu.collision()
    cu.close()
    assert not faults(fake)


def _small_list(tb, cu, dims):
    cu.forcing(markers(tb, 40, dims), ALPHA, BETA)


def _large_list(tb, cu, dims):
    cu.set_markers(markers(tb, 9000, dims, seed=2))


def _attach(tb, cu, dims, **turbine):
    rt = tb.RushtonTurbine(*dims, tip_speed=0.1, startup_steps=0, **turbine)
    d = rt.increment(1)
    cu.attach_rushton(rt, d, 0.0, d)


def _attach_small(tb, cu, dims):
    _attach(tb, cu, dims, impeller_diameter=9.0, blade_height=3.0, n_blades=2)


@pytest.mark.parametrize("first", [None, _small_list, _attach_small])
@pytest.mark.parametrize("grow", [_large_list, _attach])
def test_an_allocation_that_fails_costs_that_call_alone(fake, first, grow):
    """Every allocation of a list upload fails in turn: the call says so, and the
    calls after it -- the impeller's, a list that fits what was there before, then the
    same list again -- find every buffer in place or say that there is none."""
    dims = (48, 48, 48)
    lib = fake.load_library()
    for nth in range(1, 200):
        cu = fake.ComputeUnit(x=dims[0], y=dims[1], z=dims[2], nu=1e-3)
        cu.initialise(1.0)
        if first:
            first(fake, cu, dims)
        lib.fake_fail(nth)
        try:
            grow(fake, cu, dims)
            failed = False
        except fake.TdlbError:
            failed = True
        lib.fake_fail(0)
        if failed:
            for call in (lambda: cu.rotate_impeller(0.2, 0.1), lambda: cu.forcing_resident(ALPHA, BETA), cu.impeller_load):
                try:
                    call()
                except fake.TdlbError:
                    pass
                assert not faults(fake), f"allocation {nth}"
            for n in (40, 30):
                cu.forcing(markers(fake, n, dims), ALPHA, BETA)
                assert not faults(fake), f"allocation {nth}"
            grow(fake, cu, dims)
        cu.forcing_resident(ALPHA, BETA)
        cu.collision()
        cu.forcing_resident(ALPHA, BETA)
        assert not faults(fake), f"allocation {nth}"
        cu.close()
        if not failed:
            break
    assert nth > 1


def _ball(tb, at):
    m = np.zeros(27, tb.MARKER_DTYPE)
    for q, name in enumerate("ijk"):
        m[name] = at[q] + 3 * (np.arange(27) // 3 ** q % 3)
    return m


def test_steps_read_the_force_of_the_list_that_was_applied(fake):
    """The outer launch of a split step reads no force: it is only queued when the
    last forcing pass applied the list whose zone it leaves out."""
    lib = fake.load_library()

    def outer(step):
        n = lib.fake_launches(b"k_step_simple<float, 1, false, false, true, 1>")
        step()
        return lib.fake_launches(b"k_step_simple<float, 1, false, false, true, 1>") - n

    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3)
    cu.initialise(1.0)
    force = lambda: cu.forcing_resident(ALPHA, BETA)  # noqa: E731
    cu.set_markers(_ball(fake, (20, 30, 40)))
    force()
    cu.collision()                       # from moments
    force()
    cu.collision()
    force()
    assert outer(cu.collision) == 1
    force()
    cu.set_markers(_ball(fake, (60, 30, 40)))
    assert outer(cu.collision) == 0      # the first ball's force
    force()
    cu.collision()
    force()
    assert outer(cu.collision) == 1
    cu.forcing(_ball(fake, (10, 70, 10)), ALPHA, BETA)
    _attach(fake, cu, (96, 96, 96))
    assert outer(cu.collision) == 0      # the last ball's force
    for _ in range(2):
        force()
        cu.collision()
    force()
    assert outer(cu.collision) == 1
    # blades outside the impeller's swept volume, then inside again
    rt = fake.RushtonTurbine(96, 96, 96, tip_speed=0.1, startup_steps=0)
    inside = rt.rotating(0.1, rt.increment(1))
    outside = inside.copy()
    outside["i"] = (outside["i"] + 30) % 96
    for blades, split in ((inside, 1), (outside, 1), (inside, 0), (inside, 1), (inside, 1)):
        force()
        cu.set_rotating_markers(blades)
        n = outer(cu.collision)
        assert n <= split, "the force of blades outside the zone"
    assert n == 1
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("overlap", [None, True, "always"])
def test_a_step_follows_what_the_caller_queued_on_the_stream(fake, overlap):
    """Every launch of a step comes after the caller's own work on the handle's
    stream (a replayed graph): by itself, or after join() where split steps
    were asked for."""
    lib = fake.load_library()
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming="Esotwist")
    if overlap is not None:
        cu.set_overlap(overlap)
    cu.initialise(1.0)
    cu.set_markers(_ball(fake, (20, 30, 40)))
    cu.forcing_resident(ALPHA, BETA)
    for _ in range(4):
        cu.step(ALPHA, BETA)
    assert lib.fake_launches(b"k_step_esotwist<float, 1, false, false, true, true, 1>") > 0
    stream = cu.stream
    for _ in range(4):
        if overlap is not None:
            cu.join()
        number = lib.fake_foreign(stream)
        n = lib.fake_unordered(b"k_step_", stream, number)
        cu.step(ALPHA, BETA)
        assert lib.fake_unordered(b"k_step_", stream, number) == n, "a step launch runs beside the caller's work"
    if overlap is not None:
        before = lib.fake_launches(b"true, 1>")
        cu.step(ALPHA, BETA)
        assert lib.fake_launches(b"true, 1>") == before + 1, "asked for, steps stay split"
    cu.close()
    assert not faults(fake)


CASES = [("Simple", "fp32"), ("Esotwist", "fp32"), ("Simple", "fp16"), ("Esotwist", "bf16")]


def _loop(tb, cu, steps, rt=None):
    for s in range(steps):
        if rt is None:
            cu.rotate_impeller(0.1 * s, 0.1)
        else:
            cu.set_rotating_markers(rt.rotating(0.1 * s, 0.1))
        cu.collision()
        cu.forcing_resident(ALPHA, BETA)


@pytest.mark.parametrize("streaming,storage", CASES)
@pytest.mark.parametrize("blades", ["device", "host"])
def test_the_step_loop_allocates_nothing(fake, streaming, storage, blades):
    """After an attach, also another one on the same handle, split steps and
    residual box included. (Host blades: two pinned buffers on the first two calls.)"""
    lib = fake.load_library()
    dims = (96, 96, 96)
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
    for _ in range(2):
        _attach(fake, cu, dims)
        rt = fake.RushtonTurbine(*dims, tip_speed=0.1, startup_steps=0) if blades == "host" else None
        for q in range(2):
            if rt is not None:
                cu.set_rotating_markers(rt.rotating(0.3 * q, 0.1))
        before = lib.fake_mallocs()
        cu.initialise(1.0)
        cu.forcing_resident(ALPHA, BETA)
        _loop(fake, cu, 6, rt)
        assert lib.fake_mallocs() == before
        assert lib.fake_launches(b", 1>(") > 0, "the steps split"
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("streaming,storage", CASES)
def test_without_memory_for_the_zone_steps_do_not_split(fake, streaming, storage):
    """Each allocation of an attach fails in turn: the attach says so, or the
    steps run, split or not."""
    lib = fake.load_library()
    dims = (96, 96, 96)
    unsplit = 0
    for nth in range(1, 60):
        cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
        cu.initialise(1.0)
        before = lib.fake_mallocs()
        lib.fake_fail(nth)
        try:
            _attach(fake, cu, dims)
            lib.fake_fail(0)
            cu.forcing_resident(ALPHA, BETA)
            n = lib.fake_launches(b", 1>(")
            _loop(fake, cu, 4)
            unsplit += lib.fake_launches(b", 1>(") == n
        except fake.TdlbError:
            pass
        lib.fake_fail(0)
        cu.close()
        assert not faults(fake), f"allocation {nth}"
        if lib.fake_mallocs() - before < nth:
            break
    assert unsplit == (storage == "fp32")   # (with a residual box the zone is asked for twice)


def _zone_builds(tb):
    return tb.load_library().fake_launches(b"k_zone_words")


@pytest.mark.parametrize("streaming,storage", CASES)
@pytest.mark.parametrize("order", ["before", "after", "list"])
def test_markers_that_change_every_step_have_no_zone(fake, streaming, storage, order):
    """A zone is planned for a list that stays, not for each list of a geometry that
    is set anew before or after the collision, or handed to forcing()."""
    lib = fake.load_library()
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
    if storage != "fp32":
        cu.set_residual_box(30, 50, 30, 50, 30, 50)
    cu.initialise(1.0)
    for s in range(6):
        ball = _ball(fake, (20 + 5 * s, 30, 40))
        if order == "before":
            cu.set_markers(ball)
        if s:
            cu.collision()
        if order == "after":
            cu.set_markers(ball)
        if order == "list":
            cu.forcing(ball, ALPHA, BETA)
        else:
            cu.forcing_resident(ALPHA, BETA)
    assert _zone_builds(fake) == 0
    if order != "list":                  # and now it stays
        waits = None
        for s in range(6):
            if s == 3:
                waits = lib.fake_waits()
            cu.step(ALPHA, BETA)
        assert _zone_builds(fake) == 1 and lib.fake_waits() == waits
        assert lib.fake_launches(b", 1>(") > 0
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("streaming,storage", CASES)
def test_blades_outside_the_zone_do_not_rebuild_it(fake, streaming, storage):
    lib = fake.load_library()
    dims = (96, 96, 96)
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
    _attach(fake, cu, dims)
    rt = fake.RushtonTurbine(*dims, tip_speed=0.1, startup_steps=0)
    cu.initialise(1.0)
    cu.forcing_resident(ALPHA, BETA)
    for s in range(10):
        blades = rt.rotating(0.1 * s, 0.1)
        if s % 5 > 1:
            blades["i"] = (blades["i"] + 30) % 96
        cu.set_rotating_markers(blades)
        if s == 4:
            waits = lib.fake_waits()
        cu.collision()
        cu.forcing_resident(ALPHA, BETA)
    assert _zone_builds(fake) == 1 and lib.fake_waits() == waits
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("streaming,storage", CASES)
@pytest.mark.parametrize("overlap", [None, False, "always"])
def test_steps_are_captured_after_the_markers_changed(fake, streaming, storage, overlap):
    """A captured step neither waits nor allocates, whatever changed before it."""
    lib = fake.load_library()
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
    if overlap is not None:
        cu.set_overlap(overlap)
    cu.initialise(1.0)
    for s in range(3):
        _attach(fake, cu, (96, 96, 96))
        if storage != "fp32" and s:
            cu.set_residual_box(30, 50 + s, 30, 50, 30, 50)
        cu.forcing_resident(ALPHA, BETA)
        for _ in range(s):
            cu.step(ALPHA, BETA)
        if s == 0 and storage == "fp32":
            cu.collision()               # (the moment form's step)
        lib.fake_capture(1)
        for _ in range(3):
            cu.rotate_impeller(0.1, 0.1)
            cu.step(ALPHA, BETA)
        lib.fake_capture(0)
        assert not faults(fake), f"after attach {s}"
    cu.close()


def test_the_impeller_load_is_captured_after_another_attach(fake):
    """The load's slots and scratch come with the impeller: no load allocates or waits."""
    lib = fake.load_library()
    dims = (48, 48, 48)
    out = np.zeros(5)
    lib.fake_pin(out.ctypes.data, out.nbytes)
    cu = fake.ComputeUnit(x=48, y=48, z=48, nu=1e-3)
    cu.initialise(1.0)
    for s in range(3):
        _attach(fake, cu, dims)
        cu.forcing_resident(ALPHA, BETA)
        before = lib.fake_mallocs()
        lib.fake_capture(1)
        cu.impeller_load_async(out.ctypes.data)
        lib.fake_capture(0)
        cu.impeller_load()
        assert lib.fake_mallocs() == before
        assert not faults(fake), f"attach {s}"
    cu.close()


@pytest.mark.parametrize("at,pinned", [(0, 40), (4, 80), (8, 48), (8, 40), (0, 8), (0, 0)])
def test_the_load_goes_to_any_address(fake, at, pinned):
    """5 doubles at an address that is no multiple of 8, or that leave the pinned
    range, are copied there; the kernel writes only what it can."""
    lib = fake.load_library()
    buf = np.zeros(16)
    if pinned:
        lib.fake_pin(buf.ctypes.data, pinned)
    cu = fake.ComputeUnit(x=48, y=48, z=48, nu=1e-3)
    cu.initialise(1.0)
    _attach(fake, cu, (48, 48, 48))
    cu.forcing_resident(ALPHA, BETA)
    cu.impeller_load_async(buf.ctypes.data + at)
    cu.close()
    assert not faults(fake)


@pytest.mark.parametrize("V", [1, 2, 4])
@pytest.mark.parametrize("words", [1, 3, 4, 17, 134217728, 134217729, 268435457, 2 ** 29, 32767 * 32767])
def test_every_listed_word_has_its_lanes(fake, V, words):
    """The inner launch: 32 / V lanes of 128-thread blocks for each of up to 2^30 words
    (x * z rows of few cells along y)."""
    lib = fake.load_library()
    lib.fake_listed_word.restype = lib.fake_listed_blocks.restype = ctypes.c_longlong
    lib.fake_listed_blocks.argtypes = [ctypes.c_longlong, ctypes.c_uint]
    blocks = lib.fake_listed_blocks(words, V)
    lanes = 32 // V
    assert blocks < 2 ** 31 and (blocks - 1) * 128 < words * lanes <= blocks * 128
    for w in {0, words // 3, words // 2, words - 1}:
        for lane in (0, lanes - 1):
            thread = w * lanes + lane
            assert lib.fake_listed_word(thread // 128, thread % 128, V) == w


@pytest.mark.parametrize("nx,ny,nz", [(3, 1, 3), (400, 400, 400), (2100, 33, 2100), (8000, 32, 8000), (32767, 2, 32767),
                                      (256, 32767, 255)])
def test_gather_items_of_the_largest_planes(fake, nx, ny, nz):
    """The batched gather's work items name every tile of planes and stencil cells."""
    out = (ctypes.c_int * 4)()
    for p0 in {0, 8, nx * nz // 16 * 8, (nx * nz - 1) // 8 * 8}:
        for j0 in {0, (ny - 1) // 32 * 32, (ny - 1) // 64 * 32}:
            fake.load_library().fake_gather_item(61, j0, p0, out)
            assert list(out) == [61, 0, j0, p0]


@pytest.mark.parametrize("streaming,storage", CASES)
def test_the_automatic_mode_comes_back_and_shows_its_zone(fake, streaming, storage):
    lib = fake.load_library()
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming, storage=storage)
    cu.initialise(1.0)
    _attach(fake, cu, (96, 96, 96))

    def split():
        n = lib.fake_launches(b", 1>(")
        cu.step(ALPHA, BETA)
        return lib.fake_launches(b", 1>(") > n

    cu.forcing_resident(ALPHA, BETA)
    with pytest.raises(fake.TdlbError):
        cu.read_zone()                   # not planned yet
    for _ in range(3):
        cu.step(ALPHA, BETA)
    assert split() and cu.read_zone().shape == (96, 96, 96)
    if storage == "fp32":                # (a boxed step has an outer launch in any mode)
        cu.set_overlap(False)
        assert not split()
        with pytest.raises(fake.TdlbError):
            cu.read_zone()
        cu.set_overlap("auto")
        assert split() and cu.read_zone().shape == (96, 96, 96)
        cu.set_cells_per_thread(2)
        assert not split()
        with pytest.raises(fake.TdlbError):
            cu.read_zone()
    for bad in (-2, 3):
        with pytest.raises(fake.TdlbError):
            cu.set_overlap(bad)
    cu.close()
    assert not faults(fake)


CX = [1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0]
CY = [0, 0, 1, -1, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1]
CZ = [0, 0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1]


@pytest.mark.parametrize("shape", [(40, 96, 36), (45, 38, 51), (17, 5, 3), (9, 2, 64), (31, 3, 30)])
@pytest.mark.parametrize("cells,es", [(128, 4), (512, 4), (128, 2), (256, 2), (1024, 2)])
@pytest.mark.parametrize("ahead", [0, 1, 61])
@pytest.mark.parametrize("eso,even", [(False, False), (True, True), (True, False)])
def test_prefetch_spans_of_the_step_kernels(fake, shape, cells, es, ahead, eso, even):
    """Every span that a block's prefetch names -- `cells` elements a block or work
    item, from `ahead` of them further on -- starts and ends on 16 bytes inside its
    plane (a multiple of 64 elements) and holds what the cells away from the faces
    pull from it."""
    lib = fake.load_library()
    lib.fake_pull_span.argtypes = [ctypes.c_int] * 7 + [ctypes.c_longlong] * 2 + [ctypes.c_void_p]
    nx, ny, nz = shape
    jp, tiles = lib.fake_row_pitch(nx, ny, nz), lib.fake_prefetch_tiles()
    total = nx * nz * jp
    plane = (total + 63) // 64 * 64
    out = np.zeros(2, np.int64)
    for e0 in range(ahead * cells, total, tiles * cells):
        e1 = e0 + tiles * cells
        e = np.arange(e0, min(e1, total))
        row, j = np.divmod(e, jp)
        i, k = np.divmod(row, nz)
        inner = (i >= 1) & (i < nx - 1) & (j >= 1) & (j < ny - 1) & (k >= 1) & (k < nz - 1)
        for d in range(19):
            size = es if d < 18 else 4
            lib.fake_pull_span(nx, ny, nz, d, size, eso, even, e0, e1, out.ctypes.data)
            lo, hi = int(out[0]), int(out[1])
            assert lo % 16 == 0 and hi % 16 == 0 and 0 <= lo <= hi <= plane * size
            if d == 18:
                src = e
            elif eso:
                sg = -1 if even else 1
                src = e + (nz * jp if sg * CX[d] > 0 else 0) + (jp if sg * CZ[d] > 0 else 0) + (1 if sg * CY[d] > 0 else 0)
            else:
                src = e - (CX[d] * nz + CZ[d]) * jp - CY[d]
            src = src[inner] * size
            assert ((src >= lo) & (src + size <= hi)).all(), d


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
def test_the_zone_holds_the_attached_blades_planes(fake, streaming):
    """Blades that the host moves to other planes before the zone is planned: the
    last pass's blades are the attached ones."""
    lib = fake.load_library()
    dims = (96, 96, 96)
    cu = fake.ComputeUnit(x=96, y=96, z=96, nu=1e-3, streaming=streaming)
    cu.set_overlap("always")
    _attach(fake, cu, dims)
    rt = fake.RushtonTurbine(*dims, tip_speed=0.1, startup_steps=0)
    cu.initialise(1.0)
    cu.forcing_resident(ALPHA, BETA)
    cu.collision()                       # from moments
    cu.forcing_resident(ALPHA, BETA)
    moved = rt.rotating(0.1, rt.increment(1))
    moved["j"] = (moved["j"] + 30) % 96
    cu.set_rotating_markers(moved)
    n = lib.fake_launches(b", 1>(")
    cu.collision()
    assert lib.fake_launches(b", 1>(") == n, "the force of the attached blades' planes"
    cu.close()
    assert not faults(fake)
