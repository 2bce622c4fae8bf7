"""Calls that fail for want of device memory, and the calls after them."""
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


def leave_free(torch, nbytes):
    """A tensor that takes all device memory but `nbytes`."""
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("n", [1000, 30_000, 100_000])
def test_call_after_a_failed_allocation(ctx, torch_cuda, n):
    """The call that could not allocate reports it; the next one runs."""
    keys, pays = po.gen_perm(n, 0x5EED1201), po.gen_uniform(n, 0x5EED1201, 1, 0, 100)
    cols = [dev(torch_cuda, keys), dev(torch_cuda, pays)]
    _, hb, probe, agg = mgv.create_count_join_1G_pipeline(ctx, n)
    for head in (hb, probe):
        head.open()
        with pytest.raises(mgv.MgvError) as e:
            mgv.Pool(ctx, 1 << 20, 1 << 20, 8)  # 32 TiB
        assert e.value.status == mgv.ENOMEM
        head.consume_columns(cols, n)
        head.close()
    assert agg.result() == po.Chain(keys, pays).probe_agg(keys, pays)
    for o in (probe, agg, hb):
        o.destroy()
