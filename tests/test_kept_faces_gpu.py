"""Faces that the projection does not write (the grid's edges, walls and the
obstacle) keep their bits, also where they are below the smallest normal number:
an addition of zero would flush them."""
import numpy as np
import pytest

from opensayal_gb300 import native
from tests.parity_cases import load_lib
from tests.test_tiles_gpu import state_of, tunnel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(256, 128), (264, 70), (257, 63), (800, 400)])
@pytest.mark.parametrize("drain", [0, 1])
@pytest.mark.parametrize("pressure", [0, 1])
@pytest.mark.parametrize("resident", [-1, 1])
def test_subnormal_faces_equal_plain(gpu, w, h, drain, pressure, resident):
    base = tunnel(w, h, projection_n=9, enable_drain=drain, enable_pressure=pressure)
    state = state_of(base, w + h)
    rng = np.random.default_rng(w)
    solid = load_lib(base, {}).download("is_solid") != 0
    for field in ("vel_x", "vel_y"):  # solid cells hold faces that nothing writes
        state[field][solid] = (rng.uniform(-1e-39, 1e-39, w * h).astype(np.float32))[solid]
    plain, tiles = base.copy(), base.copy()
    plain.projection_block = -1
    tiles.projection_block, tiles.projection_resident = 4, resident
    a, b = load_lib(plain, state), load_lib(tiles, state)
    a.run_phase(native.PHASE_PROJECTION, None, 0.05)
    b.run_phase(native.PHASE_PROJECTION, None, 0.05)
    for field in ("vel_x", "vel_y"):
        x, y = a.download(field), b.download(field)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), field
    assert (np.abs(a.download("vel_x")) < 1e-38).sum() > 0
    a.close()
    b.close()
