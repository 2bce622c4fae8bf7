"""Hash builds on both sides of every change of path: one CTA (a table of one
region), compare-and-swap, region staging with smaller and full-size regions,
and more regions than a sorted tile takes; with a filter on the build side,
reserved keys, repeated keys, keys that all fall into one region's staging
share, and a second consume into a built table.  COUNT, SUM and the table's
own counters against the oracle's chained table."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev
from querymix import make_query_columns, oracle_answer

pytestmark = pytest.mark.gpu
INT32_MIN = -(1 << 31)


def build_rows(n, kind, seed):
    if kind == "distinct":
        return po.gen_perm(n, seed)
    if kind == "repeated":
        return po.gen_uniform(n, seed, 0, 0, max(1, n // 3))
    if kind == "reserved":
        k = po.gen_perm(n, seed)
        k[::max(1, n // 50)] = INT32_MIN
        return k
    k = po.gen_perm(n, seed)  # "hot": a few thousand rows share one key
    k[:min(n // 2, 3000)] = 5
    return k


@pytest.mark.parametrize("payload", [True, False])
@pytest.mark.parametrize("kind", ["distinct", "repeated", "reserved", "hot"])
@pytest.mark.parametrize("n,lf", [(1, 0.5), (4096, 0.5), (4097, 0.5), (16384, 0.95), (65535, 0.5), (65536, 0.5),
                                  (65537, 0.95), (300007, 0.5), (1 << 20, 0.7)])
def test_build_paths(ctx, torch_cuda, n, lf, kind, payload):
    seed = 0x5EED0F01 + n + int(100 * lf)
    bk = build_rows(n, kind, seed)
    bp = po.gen_uniform(n, seed, 1, INT32_MIN, 1 << 32) if payload else np.zeros(n, np.int32)
    bf = po.gen_uniform(n, seed, 2, 0, 100)
    npb = 20011
    pk = po.gen_uniform(npb, seed, 3, 0, n + n // 8 + 1)
    pk[::101] = INT32_MIN
    pp = po.gen_uniform(npb, seed, 4, INT32_MIN, 1 << 32)
    hb = mgv.Op.hash_build(ctx, 0, 1 if payload else -1, n, lf)
    sel = mgv.Op.select(ctx, 2, 79, hb)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)
    cols = [dev(torch_cuda, c) for c in (bk, bp, bf)]
    dk, dp = dev(torch_cuda, pk), dev(torch_cuda, pp)

    def check(keys, pays):
        probe.open(); probe.consume_columns([dk, dp], npb); probe.close()
        assert agg.result() == po.Chain(keys, pays).probe_agg(pk, pp)
        info = hb.result()
        assert info.rows == len(keys)
        assert info.reserved_key_rows == int((keys == INT32_MIN).sum())
        assert info.has_duplicates == int(len(np.unique(keys)) < len(keys))

    hb.open(); hb.consume_columns(cols, n); hb.close()  # every row
    check(bk, bp)
    sel.open(); sel.consume_columns(cols, n); sel.close()  # the same operator again, filtered
    keep = bf <= 79
    check(bk[keep], bp[keep])
    cut = n // 3  # and in two parts
    hb.open()
    hb.consume_columns([c[:cut] for c in cols], cut)
    hb.consume_columns([c[cut:] for c in cols], n - cut)
    hb.close()
    check(bk, bp)
    for o in (probe, agg, sel, hb):
        o.destroy()


@pytest.mark.parametrize("radix_bits", [0, 4])
def test_build_scratch_across_a_capture(ctx, torch_cuda, radix_bits):
    """A build leaves its scratch zeroed for the next one; a captured build,
    which runs when it is replayed, neither relies on that nor claims it."""
    torch, n = torch_cuda, 150_001
    sides = [(po.gen_perm(n, 0x5EED0F61 + i), po.gen_uniform(n, 0x5EED0F61 + i, 1, 0, 1 << 20)) for i in range(2)]
    sides[1][0][::1000] = INT32_MIN
    pk, pp = po.gen_uniform(20011, 0x5EED0F63, 0, 0, n + n // 8), po.gen_uniform(20011, 0x5EED0F63, 1, 0, 1 << 20)
    cols = [[dev(torch, c) for c in side] for side in sides]
    probe_cols = [dev(torch, pk), dev(torch, pp)]
    hb = mgv.Op.hash_build(ctx, 0, 1, n, 0.5, radix_bits=radix_bits)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)

    def check(side):
        probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
        assert agg.result() == po.Chain(*side).probe_agg(pk, pp)
        assert hb.result().reserved_key_rows == int((side[0] == INT32_MIN).sum())

    def build(i):
        hb.open(); hb.consume_columns(cols[i], n); hb.close()
        check(sides[i])

    build(0)
    build(1)
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        hb.open(stream=st.cuda_stream)
        hb.consume_columns(cols[1], n, stream=st.cuda_stream)
    with torch.cuda.stream(st):
        g.replay()
    hb.close(stream=st.cuda_stream)
    check(sides[1])
    build(0)
    with torch.cuda.stream(st):
        g.replay()
    torch.cuda.synchronize()
    build(0)
    build(1)
    for o in (probe, agg, hb):
        o.destroy()


def test_build_without_room_for_staging_shares(ctx, torch_cuda):
    """With room for exact staging ranges (16 bytes a row) but not for shares
    of twice the expected rows (24), the build takes the exact ranges."""
    torch, n = torch_cuda, 1 << 24
    bk, bp = po.gen_perm(n, 0x5EED0F71), po.gen_uniform(n, 0x5EED0F71, 1, 0, 1 << 20)
    pk, pp = po.gen_uniform(50021, 0x5EED0F72, 0, 0, n + n // 8), po.gen_uniform(50021, 0x5EED0F72, 1, 0, 1 << 20)
    cols, probe_cols = [dev(torch, bk), dev(torch, bp)], [dev(torch, pk), dev(torch, pp)]
    hb = mgv.Op.hash_build(ctx, 0, 1, n, 0.5)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 20 * n, dtype=torch.uint8, device="cuda")
    hb.open()
    l0 = ctx.launches
    hb.consume_columns(cols, n)
    assert ctx.launches - l0 == 5  # histogram, scan, staging, regions, global insert
    hb.close()
    del hog
    torch.cuda.empty_cache()
    for _ in range(2):
        probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
        assert agg.result() == po.Chain(bk, bp).probe_agg(pk, pp)
        assert hb.result().rows == n and hb.result().has_duplicates == 0
        hb.open(); hb.consume_columns(cols, n); hb.close()
    for o in (probe, agg, hb):
        o.destroy()


def test_build_more_regions_than_a_tile_sorts(ctx, torch_cuda):
    """2^23 {key, payload} rows at load factor 0.2: 5120 regions."""
    n = 1 << 23
    bk, bp = po.gen_perm(n, 0x5EED0F41), po.gen_uniform(n, 0x5EED0F41, 1, 0, 1 << 20)
    pk, pp = po.gen_uniform(50021, 0x5EED0F42, 0, 0, n + n // 8), po.gen_uniform(50021, 0x5EED0F42, 1, 0, 1 << 20)
    _, hb, probe, agg = mgv.create_count_join_1G_pipeline(ctx, n, 0.2)
    hb.open(); hb.consume_columns([dev(torch_cuda, bk), dev(torch_cuda, bp)], n); hb.close()
    probe.open(); probe.consume_columns([dev(torch_cuda, pk), dev(torch_cuda, pp)], len(pk)); probe.close()
    assert agg.result() == po.Chain(bk, bp).probe_agg(pk, pp)
    assert hb.result().rows == n and hb.result().has_duplicates == 0
    for o in (probe, agg, hb):
        o.destroy()


def test_batch_tables_of_many_region_counts(ctx, torch_cuda):
    """One launch over tables of 200, 128, 100, 64, 3, 1 and 0 regions (8192
    rows each at load factor 0.5): the rank counters of a tile are replicated
    more for a smaller table, so the largest one does not need the most."""
    mix = []
    for i, regions in enumerate([200, 128, 100, 64, 3, 1, 0]):
        nb, npr = regions * 8192, 30011 + 1000 * i
        cols = make_query_columns(ctx, torch_cuda, nb, npr, 100, 0x5EED0F51 + i)
        mix.append(dict(nb=nb, npr=npr, bound=700, G=100, cols=cols))
    b = mgv.Batch(ctx, [mgv.query_desc(q["cols"][0], q["nb"], *q["cols"][1:], q["npr"], q["bound"], q["G"])
                        for q in mix], mgv.BatchConfig(0.5))
    for _ in range(2):
        b.run()
    for i, q in enumerate(mix):
        assert b.result(i) == oracle_answer(q), i
    b.destroy()
