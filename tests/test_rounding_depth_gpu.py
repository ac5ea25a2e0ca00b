"""With 16-bit storage the depth says how often fields are rounded. A depth that the
library chooses for resident forms rounds no more often than the passes that it
would choose otherwise (12 sweeps deep at this size)."""
import pytest

from opensayal_gb300 import native
from opensayal_gb300.fluid import Fluid
from tests.test_tiles_gpu import tunnel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [native.STORAGE_F16, native.STORAGE_BF16])
@pytest.mark.parametrize("n,least", [(50, 16), (20, 16), (12, 12)])
def test_chosen_depth_rounds_seldom(gpu, storage, n, least):
    with Fluid(tunnel(256, 128, projection_n=n, storage=storage)) as f:
        view = f.fields()
        if view.projection_resident:
            assert view.projection_block >= least
        else:
            assert view.projection_block >= 12
