"""The advections of open cells against the general samplers. A batch advects
by the general samplers, a tunnel of its own by open samples where cell and
sample are open: the same bits, with steps of a fraction of a cell and of many,
samples that leave the grid, cells that are not finite, each storage, odd
heights (a thread takes two rows) and grids without any open cell."""
import numpy as np
import pytest

from opensayal_gb300 import native
from opensayal_gb300.batch import Batch
from opensayal_gb300.fluid import Fluid
from tests.parity_cases import FIELDS
from tests.test_tiles_gpu import equal, state_of, tunnel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(3, 3), (5, 5), (6, 7), (33, 18), (129, 61), (257, 40)])
@pytest.mark.parametrize("d_t", [0.05, 3.0])
@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("over", [{}, {"idw_mode": 1}, {"cell_size": 2.0},
                                  {"storage": native.STORAGE_F16},
                                  {"storage": native.STORAGE_BF16}])
def test_open_samples_equal_general(gpu, w, h, d_t, wild, over):
    cfg = tunnel(w, h, projection_n=2, projection_block=2, viscosity=0.0, d_t=d_t, tunnel_smoke=1.0,
                 enable_drain=w % 2, **over)
    state = state_of(cfg, 3 * w + h, wild)
    if wild:
        at = np.random.default_rng(w).integers(0, w * h, 2)
        state["smoke"][at] = [np.nan, np.inf]
    with Batch([cfg], block_k=2) as b, Fluid(cfg) as f:
        for x in (b.scenario(0), f):
            for k, a in state.items():
                x.upload(k, a)
        b.step(2)
        b.synchronize()
        for _ in range(2):
            f.update(None, cfg.d_t)
        equal(f, b.scenario(0), FIELDS)
