"""The tile kernels at the edges of their tiles: columns around a strip's 256,
odd widths, heights around a strip, a cluster and a region, sweep counts that
leave a short last pass, and cells that are not finite. FP32 results are the
bits of the plain per-sweep kernels, 16-bit results those of the same depth
pass by pass, and a batch's those of each member alone: no tolerance."""
import numpy as np
import pytest

import oracle
from opensayal_gb300 import native
from opensayal_gb300.batch import Batch
from opensayal_gb300.fluid import Fluid, default_config
from tests.parity_cases import FIELDS, load_lib, random_state, same_bits

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (255, 65), (256, 64), (257, 63), (241, 128), (480, 129), (497, 97), (252, 511),
         (1016, 31)]


def tunnel(w, h, **over):
    c = default_config(w, h)
    c.tunnel_speed = 2.0
    c.viscosity = 0.02
    c.obstacle_radius = min(w, h) / 7.0
    for k, v in over.items():
        setattr(c, k, v)
    return c


def state_of(cfg, seed, wild=False):
    state = random_state(cfg, seed, oracle.OracleFluid(cfg).is_solid)
    if wild:
        rng = np.random.default_rng(seed)
        for field in ("vel_x", "vel_y"):
            at = rng.integers(0, cfg.width * cfg.height, 3)
            state[field][at] = [np.nan, np.inf, -3e38]
    return state


def equal(a, b, fields):
    for field in fields:
        x, y = a.download(field), b.download(field)
        assert same_bits(np.nan_to_num(x, nan=1.5), np.nan_to_num(y, nan=1.5)), field
        assert np.array_equal(np.isnan(x), np.isnan(y)), field


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("k,n", [(2, 7), (5, 11), (8, 17), (16, 33)])
@pytest.mark.parametrize("resident", [-1, 3])
@pytest.mark.parametrize("wild", [False, True])
def test_phases_equal_plain(gpu, w, h, k, n, resident, wild):
    base = tunnel(w, h, projection_n=n, enable_pressure=(w + k) % 2)
    state = state_of(base, w + h + k, wild)
    plain, tiles = base.copy(), base.copy()
    plain.projection_block = -1
    tiles.projection_block, tiles.projection_resident = k, resident
    a, b = load_lib(plain, state), load_lib(tiles, state)
    for phase in (native.PHASE_DIFFUSION, native.PHASE_PROJECTION):
        a.run_phase(phase, None, 0.05)
        b.run_phase(phase, None, 0.05)
    equal(a, b, FIELDS + (("pressure",) if base.enable_pressure else ()))
    a.close()
    b.close()


@pytest.mark.parametrize("w,h", [(2400, 2100), (3001, 1999)])
@pytest.mark.parametrize("k", [4, 16])
def test_many_tiles_equal_plain(gpu, w, h, k):
    """Enough tiles for three rounds of CTAs that share their SMs."""
    base = tunnel(w, h, projection_n=k + 2)
    state = state_of(base, 9)
    plain, tiles = base.copy(), base.copy()
    plain.projection_block = -1
    tiles.projection_block, tiles.projection_resident = k, -1
    a, b = load_lib(plain, state), load_lib(tiles, state)
    for phase in (native.PHASE_DIFFUSION, native.PHASE_PROJECTION):
        a.run_phase(phase, None, 0.05)
        b.run_phase(phase, None, 0.05)
    equal(a, b, FIELDS)
    a.close()
    b.close()


@pytest.mark.parametrize("w,h", [(257, 129), (480, 97), (1280, 300)])
@pytest.mark.parametrize("storage", [native.STORAGE_F16, native.STORAGE_BF16])
def test_16_bit_resident_equals_passes(gpu, w, h, storage):
    base = tunnel(w, h, projection_n=21, storage=storage, projection_block=8)
    state = state_of(base, 5)
    passes, resident = base.copy(), base.copy()
    passes.projection_resident, resident.projection_resident = -1, 3
    a, b = load_lib(passes, state), load_lib(resident, state)
    for _ in range(2):
        a.update(None, 0.02)
        b.update(None, 0.02)
    equal(a, b, FIELDS)
    a.close()
    b.close()


@pytest.mark.parametrize("block_k", [1, 4, 12, 16])
def test_batch_members_equal_alone(gpu, block_k):
    cfgs = []
    for i, (w, h) in enumerate([(8, 8), (255, 127), (256, 128), (257, 129), (241, 200), (33, 400),
                                (600, 113), (64, 257), (320, 144), (96, 145)]):
        c = tunnel(w, h, projection_n=2 * block_k + 1 + i, projection_block=block_k)
        c.storage = (native.STORAGE_F32, native.STORAGE_F16, native.STORAGE_BF16)[i % 3]
        if i == 4:
            c.viscosity = 0.0
        cfgs.append(c)
    states = [state_of(c, 40 + i) for i, c in enumerate(cfgs)]
    with Batch(cfgs, block_k=block_k) as b:
        for i, st in enumerate(states):
            for k, a in st.items():
                b.scenario(i).upload(k, a)
        b.step(2)
        b.synchronize()
        for i, (c, st) in enumerate(zip(cfgs, states)):
            with Fluid(c) as f:
                for k, a in st.items():
                    f.upload(k, a)
                for _ in range(2):
                    f.update(None, c.d_t)
                equal(f, b.scenario(i), FIELDS)
