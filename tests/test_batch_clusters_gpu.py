"""A batch whose tiles change with its members: many low tunnels (clusters of two
CTAs), a tall one that joins (four), and leaves again (two). Members advance as
alone all the while."""
import pytest

from opensayal_gb300 import native
from opensayal_gb300.batch import Batch
from tests.parity_cases import FIELDS, load_lib
from tests.test_resident_order_gpu import assert_same
from tests.test_tiles_gpu import state_of, tunnel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_k", [2, 8, 16])
def test_members_equal_alone_while_tiles_change(gpu, block_k):
    low = []
    for i in range(120):
        c = tunnel(20 + 37 * i % 300, (8, 33, 65, 71, 72, 64)[i % 6], projection_block=block_k,
                   projection_n=block_k + i % 7)
        c.storage = (native.STORAGE_F32, native.STORAGE_BF16)[i % 2]
        low.append(c)
    tall = tunnel(130, 301, projection_n=21, projection_block=block_k)
    watched = [0, 1, 2, 3, 4, 5, 7, 64, 119]
    states = {i: state_of(low[i], i) for i in watched}
    tall_state = state_of(tall, 99)
    with Batch.dynamic(block_k=block_k, budget_bytes=1 << 28) as b:
        ids = [b.add(c, -1) for c in low]
        for i in watched:
            for k, a in states[i].items():
                b.scenario(ids[i]).upload(k, a)
        b.step(1)
        t = b.add(tall, -1)
        for k, a in tall_state.items():
            b.scenario(t).upload(k, a)
        b.step(2)
        b.synchronize()
        with load_lib(tall, tall_state) as f:
            for _ in range(2):
                f.update(None, tall.d_t)
            assert_same(f, b.scenario(t), FIELDS)
        b.remove(t)
        b.step(1)
        b.synchronize()
        for i in watched:
            with load_lib(low[i], states[i]) as f:
                for _ in range(4):
                    f.update(None, low[i].d_t)
                assert_same(f, b.scenario(ids[i]), FIELDS)
