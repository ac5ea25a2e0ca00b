"""What the host decides for the tile phases, read from the launches that a step
makes: no GPU needed."""
import pytest

from opensayal_gb300 import native
from tests.host_only import DIFFUSE, PROJECT, Handle, launches, load, tunnel


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
