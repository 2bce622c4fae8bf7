"""Rows materialised by a sink: the staged rows of a warp are written out in
blocks that may span many small pool buffers, with and without a select or a
probe in front, and with rows that have many matches."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev, sorted_rows

pytestmark = pytest.mark.gpu


def read_sink(torch, sink, ncols):
    rows = sink.result()
    out = [torch.empty(max(rows, 1), dtype=torch.int32, device="cuda") for _ in range(ncols)]
    for c in range(ncols):
        assert sink.sink_read(c, out[c].data_ptr(), rows) == rows
    return [o.cpu().numpy()[:rows] for o in out]


@pytest.mark.parametrize("payload", [True, False])
@pytest.mark.parametrize("keys", ["distinct", "repeated", "reserved"])
@pytest.mark.parametrize("n,capacity", [(1, 128), (127, 128), (129, 128), (511, 256), (513, 128), (6145, 128),
                                        (100003, 4096)])
def test_join_to_sink(ctx, torch_cuda, n, capacity, keys, payload):
    """Every match of the oracle's chained join, for unique tables, tables with
    up to 12 rows a key, and a table whose reserved key INT32_MIN repeats."""
    nb = 3000
    bk = po.gen_perm(nb, 0x5EED0C01)
    if keys == "repeated":
        bk = (bk % 250).astype(np.int32)
    if keys == "reserved":
        bk[:7] = -(1 << 31)
    bp = po.gen_uniform(nb, 0x5EED0C01, 1, -(1 << 31), 1 << 32) if payload else np.zeros(nb, np.int32)
    pk = po.gen_uniform(n, 0x5EED0C02, 0, 0, 300 if keys == "repeated" else 4000)
    if keys == "reserved":
        pk[::max(1, n // 40)] = -(1 << 31)
    pp = np.arange(n, dtype=np.int32)
    want = po.Chain(bk, bp).probe_emit(pk, pp)
    hb = mgv.Op.hash_build(ctx, 0, 1 if payload else -1, nb)
    hb.open(); hb.consume_columns([dev(torch_cuda, bk), dev(torch_cuda, bp)], nb); hb.close()
    pool = mgv.Pool(ctx, max(1, -(-len(want) // capacity)), capacity, 3)
    sink = mgv.Op.sink(ctx, pool)
    probe = mgv.Op.hash_probe(ctx, 0, hb, sink)
    for _ in range(2):  # reopening returns the buffers
        probe.open(); probe.consume_columns([dev(torch_cuda, pk), dev(torch_cuda, pp)], n); probe.close()
        key, row, pay = read_sink(torch_cuda, sink, 3)
        assert np.array_equal(sorted_rows([key, pay, row]), sorted_rows([want[:, 0], want[:, 1], want[:, 2]]))
    for o in (probe, sink, hb):
        o.destroy()
    pool.destroy()


@pytest.mark.parametrize("select", [True, False])
@pytest.mark.parametrize("n,capacity", [(1, 128), (128, 128), (512, 128), (6145, 128), (50001, 1024)])
def test_columns_to_sink(ctx, torch_cuda, n, capacity, select):
    """[select ->] sink keeps whole rows of three columns."""
    cols = [po.gen_uniform(n, 0x5EED0C03, c, -1000, 2000) for c in range(3)]
    keep = cols[1] <= 100 if select else np.ones(n, bool)
    pool = mgv.Pool(ctx, max(1, -(-int(keep.sum()) // capacity)), capacity, 3)
    sink = mgv.Op.sink(ctx, pool)
    head = mgv.Op.select(ctx, 1, 100, sink) if select else sink
    head.open(); head.consume_columns([dev(torch_cuda, c) for c in cols], n); head.close()
    got = read_sink(torch_cuda, sink, 3)
    assert np.array_equal(sorted_rows(got), sorted_rows([c[keep] for c in cols]))
    for o in ([head, sink] if select else [sink]):
        o.destroy()
    pool.destroy()
