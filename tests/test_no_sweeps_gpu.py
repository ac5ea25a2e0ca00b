"""projection_n = 0: a step is forces, extrapolation and advection, in every form
of the projection the same bits as with the plain kernels."""
import pytest

from opensayal_gb300 import native
from opensayal_gb300.batch import Batch
from tests.parity_cases import FIELDS, load_lib
from tests.test_resident_order_gpu import assert_same
from tests.test_tiles_gpu import state_of, tunnel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,resident", [(0, 0), (1, -1), (8, -1), (8, 3)])
@pytest.mark.parametrize("viscosity", [0.0, 0.02])
@pytest.mark.parametrize("storage", [native.STORAGE_F32, native.STORAGE_BF16])
def test_step_without_sweeps_equals_plain(gpu, k, resident, viscosity, storage):
    base = tunnel(300, 130, projection_n=0, viscosity=viscosity, storage=storage,
                  enable_pressure=k == 8)
    state = state_of(base, 11)
    plain, form = base.copy(), base.copy()
    plain.projection_block = -1
    form.projection_block, form.projection_resident = k, resident
    a, b = load_lib(plain, state), load_lib(form, state)
    for _ in range(3):
        a.update(None, 0.05)
        b.update(None, 0.05)
    assert_same(a, b, FIELDS + (("pressure",) if base.enable_pressure else ()))
    a.close()
    b.close()


def test_batch_without_sweeps_equals_alone(gpu):
    cfg = tunnel(300, 130, projection_n=0)
    state = state_of(cfg, 11)
    with Batch([cfg, tunnel(96, 64, projection_n=9)], block_k=4) as batch:
        f = load_lib(cfg, state)
        for k, a in state.items():
            batch.scenario(0).upload(k, a)
        batch.step(2)
        batch.synchronize()
        for _ in range(2):
            f.update(None, cfg.d_t)
        assert_same(f, batch.scenario(0), FIELDS)
        f.close()
