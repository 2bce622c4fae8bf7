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


@pytest.mark.parametrize("radix_bits", [0, 4])
def test_replay_after_the_scratch_grew(ctx, torch_cuda, radix_bits):
    """A graph of a build keeps the scratch that it was captured with when a larger build takes a larger one."""
    torch, sizes = torch_cuda, (100_003, 2_000_003)
    sides = [(po.gen_perm(n, 0x5EED1402 + i), po.gen_uniform(n, 0x5EED1402 + i, 1, 0, 100)) for i, n in enumerate(sizes)]
    cols = [[dev(torch, c) for c in side] for side in sides]
    pk, pp = po.gen_uniform(20011, 0x5EED1404, 0, 0, 150_000), po.gen_uniform(20011, 0x5EED1404, 1, 0, 100)
    probe_cols = [dev(torch, pk), dev(torch, pp)]
    hb = mgv.Op.hash_build(ctx, 0, 1, sizes[1], radix_bits=radix_bits)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)

    def check(i):
        assert hb.result().rows == sizes[i]
        probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
        assert agg.result() == po.Chain(*sides[i]).probe_agg(pk, pp)

    def build(i):
        hb.open(); hb.consume_columns(cols[i], sizes[i]); hb.close()
        check(i)

    build(0)  # allocates, which a capture may not
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        hb.open(stream=st.cuda_stream)
        hb.consume_columns(cols[0], sizes[0], stream=st.cuda_stream)
    with torch.cuda.stream(st):
        g.replay()
    hb.close(stream=st.cuda_stream)
    check(0)
    build(1)
    other = torch.full((64 << 20,), 7, dtype=torch.int32, device="cuda")  # takes what a freed scratch would leave
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        g.replay()
    torch.cuda.synchronize()
    assert bool((other == 7).all())
    build(1)
    for o in (probe, agg, hb):
        o.destroy()
