"""Resident phases where the order between their tiles is what counts: few sweeps
(no exchange, an even number of passes), a sweep more than lie between two
exchanges, and 16-bit storage whose roundings come more often than exchanges.
The bits of the same depth pass by pass: no tolerance."""
import numpy as np
import pytest

from opensayal_gb300 import native
from opensayal_gb300.batch import Batch
from tests.parity_cases import FIELDS, load_lib
from tests.test_tiles_gpu import state_of, tunnel

pytestmark = pytest.mark.gpu


def assert_same(a, b, fields):
    """Equal cell for cell: infinities and the largest numbers apart, NaN with
    NaN, +0 with -0."""
    for field in fields:
        assert np.array_equal(a.download(field), b.download(field), equal_nan=True), field


@pytest.mark.parametrize("w,h", [(333, 187), (571, 157), (800, 400), (1003, 300)])
@pytest.mark.parametrize("k,n", [(2, 3), (2, 8), (4, 6), (4, 13), (4, 33), (6, 21), (8, 16),
                                 (8, 21), (12, 25)])
@pytest.mark.parametrize("storage", [native.STORAGE_F32, native.STORAGE_F16, native.STORAGE_BF16])
def test_resident_equals_passes(gpu, w, h, k, n, storage):
    base = tunnel(w, h, projection_n=n, storage=storage, projection_block=k,
                  enable_pressure=(w + n) % 2)
    state = state_of(base, w + k + n)
    passes, resident = base.copy(), base.copy()
    passes.projection_resident, resident.projection_resident = -1, 3
    a, b = load_lib(passes, state), load_lib(resident, state)
    assert b.fields().projection_resident == (3 if k % 4 == 0 else 1)
    for phase in (native.PHASE_DIFFUSION, native.PHASE_PROJECTION):
        a.run_phase(phase, None, 0.05)
        b.run_phase(phase, None, 0.05)
    for _ in range(2):
        a.update(None, 0.02)
        b.update(None, 0.02)
    assert_same(a, b, FIELDS + (("pressure",) if base.enable_pressure else ()))
    a.close()
    b.close()


@pytest.mark.parametrize("w,h", [(257, 63), (252, 511), (480, 129), (800, 400)])
@pytest.mark.parametrize("k,n", [(4, 33), (8, 17)])
@pytest.mark.parametrize("resident", [-1, 3])
def test_wild_states_equal_plain(gpu, w, h, k, n, resident):
    """Cells that are not finite: infinities stay apart from the largest numbers."""
    base = tunnel(w, h, projection_n=n, enable_pressure=w % 2)
    state = state_of(base, w + h + k, wild=True)
    plain, tiles = base.copy(), base.copy()
    plain.projection_block = -1
    tiles.projection_block, tiles.projection_resident = k, resident
    a, b = load_lib(plain, state), load_lib(tiles, state)
    assert b.fields().projection_resident == max(resident, 0)
    for phase in (native.PHASE_DIFFUSION, native.PHASE_PROJECTION):
        a.run_phase(phase, None, 0.05)
        b.run_phase(phase, None, 0.05)
    assert_same(a, b, FIELDS + (("pressure",) if base.enable_pressure else ()))
    a.close()
    b.close()


@pytest.mark.parametrize("k,n", [(4, 7), (8, 16), (8, 50)])
def test_resident_beside_other_work_equals_alone(gpu, k, n):
    """Other streams hold SMs meanwhile, so that a resident launch's tiles do not
    all start together: a tunnel pass by pass and a batch."""
    res = tunnel(800, 400, projection_n=n, projection_block=k, projection_resident=3)
    other = tunnel(1003, 771, projection_n=20, projection_block=8, projection_resident=-1)
    low = [tunnel(96 + 16 * i, 64 + 8 * i, projection_n=30) for i in range(6)]
    state, other_state = state_of(res, 1), state_of(other, 2)
    steps = 40
    with load_lib(res, state) as a, load_lib(res, state) as b, load_lib(other, other_state) as o, \
            Batch(low, block_k=8) as batch:
        assert a.fields().projection_resident == 3
        a.update_async(None, 0.02, steps)
        a.synchronize()
        for _ in range(steps // 8):
            o.update_async(None, 0.02, 8)
            batch.step(8)
            b.update_async(None, 0.02, 8)
        for x in (b, o, batch):
            x.synchronize()
        assert_same(a, b, FIELDS)
        with load_lib(other, other_state) as alone:
            alone.update_async(None, 0.02, steps)
            alone.synchronize()
            assert_same(o, alone, FIELDS)
