"""Probes of a table without a free slot (as many rows as slots, which a build
accepts): no run of such a table meets an empty slot, so a probe ends where its
run began, having seen every bucket once."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev, sorted_rows

pytestmark = pytest.mark.gpu


def full_table(ctx, torch, buckets, payload, dups, radix_bits):
    """(hash build, keys, payloads) of a table of about `buckets` buckets with every slot taken."""
    slots = 4 if payload else 8
    hb = mgv.Op.hash_build(ctx, 0, 1 if payload else -1, buckets * slots // 2, 0.5, radix_bits=radix_bits)
    hb.open(); hb.close()
    n = hb.result().nbuckets * slots
    keys = po.gen_perm(n, 0x5EED1501)
    if dups:
        keys = (keys // 2).astype(np.int32)
    pays = po.gen_uniform(n, 0x5EED1501, 1, -(1 << 31), 1 << 32) if payload else np.zeros(n, np.int32)
    hb.open(); hb.consume_columns([dev(torch, keys), dev(torch, pays)], n); hb.close()
    assert hb.result().rows == n and hb.result().has_duplicates == int(dups)
    return hb, keys, pays


@pytest.mark.parametrize("kernel", [3, 2, 1])
@pytest.mark.parametrize("radix_bits", [0, 2])
@pytest.mark.parametrize("payload", [True, False])
@pytest.mark.parametrize("dups", [True, False])
@pytest.mark.parametrize("buckets", [1, 2, 3, 37, 300])
def test_probe_of_a_full_table(ctx, torch_cuda, buckets, dups, payload, radix_bits, kernel):
    hb, keys, pays = full_table(ctx, torch_cuda, buckets, payload, dups, radix_bits)
    chain = po.Chain(keys, pays)
    pk = po.gen_uniform(5010, 0x5EED1502, 0, 0, len(keys) + 3)
    pp = po.gen_uniform(5010, 0x5EED1502, 1, -(1 << 31), 1 << 32)
    dk, dp = dev(torch_cuda, pk), dev(torch_cuda, pp)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)
    old = ctx.tuning()
    ctx.set_tuning(probe_kernel=kernel)
    try:
        for off in (0, 1, 4, 7):
            for n in (1, 1500, 5000):
                probe.open(); probe.consume_columns([dk[off:], dp[off:]], n); probe.close()
                assert agg.result() == chain.probe_agg(pk[off:off + n], pp[off:off + n]), (off, n)
    finally:
        ctx.set_tuning(probe_kernel=old.probe_kernel)
        for o in (probe, agg, hb):
            o.destroy()


@pytest.mark.parametrize("payload", [True, False])
@pytest.mark.parametrize("dups", [True, False])
@pytest.mark.parametrize("buckets", [1, 2, 37, 300])
def test_chain_over_a_full_table(ctx, torch_cuda, buckets, dups, payload):
    """select -> probe -> aggregate, -> group-by, and probe -> sink."""
    hb, keys, pays = full_table(ctx, torch_cuda, buckets, payload, dups, 0)
    n = 3001
    pk = po.gen_uniform(n, 0x5EED1503, 0, 0, len(keys) + 3)
    pf, pg = po.gen_uniform(n, 0x5EED1503, 1, 0, 100), po.gen_uniform(n, 0x5EED1503, 2, 0, 50)
    cols = [dev(torch_cuda, c) for c in (pk, pf, pg)]
    keep = pf <= 59
    want = po.Chain(keys, pays).probe_emit(pk, np.arange(n, dtype=np.int32))  # (key, payload, probe row)
    kept = want[keep[want[:, 2]]]
    agg, gb = mgv.Op.aggregate(ctx, 3, -1), mgv.Op.groupby(ctx, 2, 3, 50)
    for term in (agg, gb):
        probe = mgv.Op.hash_probe(ctx, 0, hb, term)
        sel = mgv.Op.select(ctx, 1, 59, probe)
        sel.open(); sel.consume_columns(cols, n); sel.close()
        sel.destroy(); probe.destroy()
    assert agg.result() == (len(kept), int(kept[:, 1].astype(np.int64).sum()))
    group = pg[kept[:, 2]]
    assert gb.result() == [(int(g), int(kept[group == g, 1].astype(np.int64).sum()), int((group == g).sum()))
                           for g in np.unique(group)]
    pool = mgv.Pool(ctx, max(1, -(-len(want) // 1024)), 1024, 4)
    sink = mgv.Op.sink(ctx, pool)
    probe = mgv.Op.hash_probe(ctx, 0, hb, sink)
    probe.open(); probe.consume_columns(cols, n); probe.close()
    assert sink.result() == len(want)
    out = [torch_cuda.empty(max(1, len(want)), dtype=torch_cuda.int32, device="cuda") for _ in range(4)]
    for c in range(4):
        sink.sink_read(c, out[c].data_ptr(), len(want))
    got = [o.cpu().numpy()[:len(want)] for o in out]
    rows = want[:, 2]
    assert np.array_equal(sorted_rows(got), sorted_rows([want[:, 0], pf[rows], pg[rows], want[:, 1]]))
    for o in (probe, sink, agg, gb, hb):
        o.destroy()
    pool.destroy()
