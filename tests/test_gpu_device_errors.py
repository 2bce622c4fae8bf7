"""A device error is reported once, by the first call that waits for it."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sync_first", [True, False])
@pytest.mark.parametrize("room,n", [(1000, 4096), (20_000, 60_000), (70_000, 200_000)])
def test_full_table_is_reported_once(ctx, torch_cuda, room, n, sync_first):
    """More rows than the table has slots, by each build path: ENOMEM from the wait that comes first, OK afterwards,
    with the rows that the table did take."""
    keys = po.gen_perm(n, 0x5EED1301)
    cols = [dev(torch_cuda, keys), dev(torch_cuda, np.arange(n, dtype=np.int32))]
    hb = mgv.Op.hash_build(ctx, 0, 1, room, 0.95)
    for _ in range(2):
        hb.open()
        hb.consume_columns(cols, n)
        if sync_first:
            with pytest.raises(mgv.MgvError) as e:
                ctx.sync()
            assert e.value.status == mgv.ENOMEM
            assert hb.try_close() == mgv.OK
            assert hb.result().rows == 4 * hb.result().nbuckets
        else:
            assert hb.try_close() == mgv.ENOMEM
        ctx.sync()
    hb.destroy()
