"""Memory that the device may still write: it outlives the work on it."""
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 30_000, 150_001])
def test_open_build_destroyed_before_its_work_ran(ctx, torch_cuda, n):
    """Destroying an open build waits for its kernels, on whatever stream they are: they write into its memory, pinned
    memory included."""
    torch = torch_cuda
    cols = [dev(torch, po.gen_perm(n, 0x5EED1401)), dev(torch, po.gen_uniform(n, 0x5EED1401, 1, 0, 100))]
    a = torch.ones((8192, 8192), dtype=torch.float32, device="cuda")
    st = torch.cuda.Stream()
    hb = mgv.Op.hash_build(ctx, 0, 1, n)
    hb.open(); hb.consume_columns(cols, n); hb.close()  # its scratch is there
    torch.cuda.synchronize()
    hb.open(stream=st.cuda_stream)
    with torch.cuda.stream(st):
        for _ in range(4):
            a = a @ a * 1e-4  # tens of milliseconds ahead of the build
    hb.consume_columns(cols, n, stream=st.cuda_stream)
    assert not st.query()
    hb.destroy()
    assert st.query()
