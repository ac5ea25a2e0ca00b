"""What the host decides for the tile phases, read from the launches that a step
makes: no GPU needed."""
import ctypes as C
import re

import pytest

from opensayal_gb300 import native
from tests.conftest import ROOT
from tests.host_only import (BATCH_DIFFUSE, BATCH_PROJECT, DIFFUSE, PROJECT, Handle, launches,
                             load, segments, tunnel)


@pytest.fixture(scope="module")
def lib():
    return load()


@pytest.mark.parametrize("w,h", [(256, 128), (333, 187), (640, 448), (1280, 720), (1920, 1080)])
@pytest.mark.parametrize("k", [2, 4, 8, 12])
@pytest.mark.parametrize("resident", [-1, 3])
@pytest.mark.parametrize("storage", [native.STORAGE_F32, native.STORAGE_BF16])
def test_no_launch_stores_to_the_copy_it_loads(lib, w, h, k, resident, storage):
    """A tile stores its cells when it is done, and nothing orders that behind
    the loads of its neighbours' halos: so a launch takes one copy of the fields
    and leaves the other, whatever n and the depth are, and the next launch
    takes what it left."""
    for n in [*range(1, 21), 33, 50]:
        cfg = tunnel(w, h, projection_n=n, projection_block=k, projection_resident=resident,
                     storage=storage)
        with Handle(lib, cfg) as f:
            assert f.update() == native.OS_OK
            tiles = launches(lib, DIFFUSE, PROJECT)
            assert tiles
            live = f.fields().vel_x
            for x in tiles:
                assert x.ui == live and x.uo != x.ui, (n, x.kind)
                live = x.uo
            live = f.fields().vel_y
            for x in tiles:
                if x.kind == PROJECT:
                    assert x.vi == live and x.vo != x.vi, n
                    live = x.vo


@pytest.mark.parametrize("w,h", [(333, 187), (571, 157), (640, 448), (800, 400), (1003, 771),
                                 (1280, 720), (1920, 1080)])
@pytest.mark.parametrize("k", [2, 4, 6, 8, 12])
@pytest.mark.parametrize("storage", [native.STORAGE_F32, native.STORAGE_F16, native.STORAGE_BF16])
def test_exchanges_lie_a_halo_of_messages_apart(lib, w, h, k, storage):
    """Packets are written again two exchanges later, and a copy is safe then
    because the messages between two exchanges go from strip to strip over a
    whole halo; the halo lasts for the sweeps between them; 16-bit fields are
    rounded after every K sweeps, whatever lies between exchanges."""
    exchanged = 0
    for n, pressure in [(9, 0), (21, 1), (50, 0), (100, 1)]:
        cfg = tunnel(w, h, projection_n=n, projection_block=k, projection_resident=3,
                     storage=storage, enable_pressure=pressure)
        with Handle(lib, cfg) as f:
            assert f.update() == native.OS_OK
            for x in launches(lib, DIFFUSE, PROJECT):
                reach = x.halo // x.R + 1
                done = since = messages = exchanges = 0
                for sweeps, sent, rounded, exchange in segments(lib, x, storage):
                    wide = storage == native.STORAGE_F32
                    assert bool(rounded) == (not wide and done > 0 and done % k == 0)
                    if exchange:
                        assert x.cooperative and messages >= reach
                        since = messages = 0
                        exchanges += 1
                    done, since, messages = done + sweeps, since + sweeps, messages + sent
                    if x.tiles > 1:
                        assert since * (2 if x.kind == PROJECT else 1) <= x.halo
                assert done == x.n
                assert x.tiles == 1 or exchanges == (x.n + x.D - 1) // x.D - 1
                exchanged += exchanges
    assert exchanged


@pytest.mark.parametrize("k,resident", [(-1, -1), (0, 0), (0, -1), (0, 3), (1, -1), (8, -1), (8, 3),
                                        (24, -1), (32, 3)])
@pytest.mark.parametrize("viscosity", [0.0, 0.02])
@pytest.mark.parametrize("pressure", [0, 1])
def test_no_sweeps_are_no_launches(lib, k, resident, viscosity, pressure):
    """projection_n = 0 is a valid step without diffusion and projection."""
    cfg = tunnel(640, 448, projection_n=0, projection_block=k, projection_resident=resident,
                 viscosity=viscosity, enable_pressure=pressure)
    with Handle(lib, cfg) as f:
        assert f.update() == native.OS_OK, lib.os_last_error()
        done = launches(lib)
        assert done and not [x for x in done if x.kind in (DIFFUSE, PROJECT)]
        for phase in (native.PHASE_DIFFUSION, native.PHASE_PROJECTION):
            assert lib.os_run_phase(f.h, phase, None, 0.05) == native.OS_OK
        assert not launches(lib)


def test_limits_of_kernels_are_never_lowered(lib):
    """A kernel's shared-memory limit is the process's, not a launch's: a handle
    that lowers it takes it from another thread's launch."""
    sizes = [(256, 128), (1920, 1080), (333, 187), (4096, 4096), (640, 448), (800, 400)]
    for resident in (-1, 3):
        for pressure in (0, 1):
            for w, h in sizes + sizes[::-1]:
                cfg = tunnel(w, h, projection_n=20, projection_block=4,
                             projection_resident=resident, enable_pressure=pressure)
                with Handle(lib, cfg) as f:
                    assert f.update() == native.OS_OK
                    assert all(x.smem <= x.limit for x in launches(lib, DIFFUSE, PROJECT))
    assert lib.state.limits_lowered == 0


def test_a_failed_query_is_made_again(tmp_path):
    """A passing error must not keep the process's later handles off the tiles."""
    lib = load(copy_to=tmp_path)  # a library without answers kept from other tests
    cfg = tunnel(640, 448, projection_n=20, projection_block=8, projection_resident=3)
    lib.state.fail_attribute = 1 << 30
    with Handle(lib, cfg) as f:
        assert f.fields().projection_resident == 0
    lib.state.fail_attribute = 0
    with Handle(lib, cfg) as f:
        assert f.fields().projection_resident == 3
        assert f.update() == native.OS_OK


def test_a_wait_that_gave_up_in_a_member_alone_is_reported(lib):
    """Members of a batch with a memory budget have no mapped word of their own; a
    step enqueued on one by itself still has to report a wait that gave up."""
    batch, mid, h = C.c_void_p(), C.c_int64(), C.c_void_p()
    assert lib.os_batch_create_dynamic(0, 4, 1 << 28, C.byref(batch)) == native.OS_OK
    cfg = tunnel(333, 187, projection_n=9)
    assert lib.os_batch_add(batch, C.byref(cfg), -1, C.byref(mid)) == native.OS_OK
    assert lib.os_batch_scenario(batch, mid, C.byref(h)) == native.OS_OK
    launches(lib)
    assert lib.os_update(h, None, 0.05) == native.OS_OK
    word = C.c_int32.from_address(launches(lib, PROJECT)[0].err)
    for call in (lambda: lib.os_synchronize(h), lambda: lib.os_update(h, None, 0.05),
                 lambda: lib.os_query(h, C.byref(C.c_int32()))):
        word.value = 1
        assert call() == native.OS_ERR_TIMEOUT
        assert word.value == 0
        assert call() == native.OS_OK
    lib.os_batch_destroy(batch)


def test_memory_of_the_exchange_is_counted_and_may_be_refused(lib):
    """Tiles that exchange hold packets: 24 bytes a cell for the projection and 16
    for the diffusion. They count as the handle's device memory, and without room
    for them the phases run pass by pass."""
    cfg = tunnel(800, 400, projection_n=50, projection_block=8, projection_resident=3)

    def member_bytes(c):
        batch, used, budget = C.c_void_p(), C.c_uint64(), C.c_uint64()
        assert lib.os_batch_create(C.byref(c), 1, 8, C.byref(batch)) == native.OS_OK
        assert lib.os_batch_memory(batch, C.byref(used), C.byref(budget)) == native.OS_OK
        lib.os_batch_destroy(batch)
        return used.value

    passes = cfg.copy()
    passes.projection_resident = -1
    packets = (24 + 16) * 800 * 400
    extra = member_bytes(cfg) - member_bytes(passes)
    assert packets <= extra <= packets + 4096
    lib.state.fail_malloc_from = packets
    try:
        with Handle(lib, cfg) as f:
            assert f.fields().projection_resident == 0
            assert f.update() == native.OS_OK
            assert all(not x.cooperative for x in launches(lib, DIFFUSE, PROJECT))
    finally:
        lib.state.fail_malloc_from = 0


@pytest.mark.parametrize("pdl", [None, "0", "1"])
def test_programmatic_launch_can_be_turned_off(lib, monkeypatch, pdl):
    """OPENSAYAL_GB300_PDL=0 turns it off for a handle and for a batch."""
    if pdl is None:
        monkeypatch.delenv("OPENSAYAL_GB300_PDL", raising=False)
    else:
        monkeypatch.setenv("OPENSAYAL_GB300_PDL", pdl)
    cfg = tunnel(333, 187, projection_n=9, projection_block=4, projection_resident=-1)
    with Handle(lib, cfg) as f:
        assert f.update() == native.OS_OK
        assert {x.pdl for x in launches(lib)} == {int(pdl != "0")}
    batch = C.c_void_p()
    assert lib.os_batch_create(C.byref(cfg), 1, 4, C.byref(batch)) == native.OS_OK
    made = launches(lib)  # the member's set-up, and the step that the graph captures
    lib.os_batch_destroy(batch)
    step = [x.pdl for x in made if x.kind in (BATCH_DIFFUSE, BATCH_PROJECT)]
    assert step and set(step) == {int(pdl != "0")}
    assert any(x.pdl for x in made) == (pdl != "0")


def test_batch_tiles_follow_the_members(lib):
    """Many members no taller than two CTAs' rows take clusters of two, few of them
    and taller ones clusters of four; a member that comes later changes it."""
    low, tall = tunnel(60, 50, projection_n=9), tunnel(60, 200, projection_n=9)

    def clusters():
        return {x.cluster for x in launches(lib, BATCH_DIFFUSE, BATCH_PROJECT)}

    for cfgs, want in (([low] * 16, 4), ([low] * 200, 2), ([low] * 200 + [tall], 4)):
        batch = C.c_void_p()
        arr = (native.OsConfig * len(cfgs))(*cfgs)
        assert lib.os_batch_create(arr, len(cfgs), 4, C.byref(batch)) == native.OS_OK
        assert clusters() == {want}
        lib.os_batch_destroy(batch)
    batch, mid = C.c_void_p(), C.c_int64()
    assert lib.os_batch_create_dynamic(0, 4, 0, C.byref(batch)) == native.OS_OK
    for members, cfg, want in ((16, low, {4}), (184, low, {2}), (1, tall, {4}), (1, low, set())):
        for _ in range(members):
            assert lib.os_batch_add(batch, C.byref(cfg), -1, C.byref(mid)) == native.OS_OK
        launches(lib)
        assert lib.os_batch_step(batch, 1, None) == native.OS_OK
        assert clusters() == want
    lib.os_batch_destroy(batch)


def test_tile_kernels_check_their_clusters():
    """Each kernel that sends messages between CTAs asks whether the launch has its
    clusters before it sends the first."""
    for name, kernels in (("os_tile.cuh", 2), ("os_tile_batch.cu", 2), ("os_tile_host.cuh", 1)):
        text = (ROOT / "opensayal_gb300" / "csrc" / name).read_text()
        opened = [m.start() for m in re.finditer(r"Link<\d> link = open_link<", text)]
        assert len(opened) == kernels, name
        for at in opened:
            asked = re.compile(r"cluster_wait\(\);[^\n]*\n  if \(!clusters_of\([^)]*\)\) return;")
            found = asked.search(text, at)
            sent = re.compile(r"(tile_sweeps|jacobi_sweeps|idle_messages)(<[^>]*>)?\(").search(text, at)
            assert found and sent and found.start() < sent.start(), name
