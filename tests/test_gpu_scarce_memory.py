"""Calls that fail for want of device memory, and the calls after them."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev
from querymix import make_query_columns, oracle_answer

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


@pytest.mark.parametrize("then", ["smaller", "same", "nothing"])
def test_build_after_a_failed_consume(ctx, torch_cuda, then):
    """A first consume without room for its scratch leaves the table to be cleared by the next one, or by the close:
    neither an earlier build's rows nor its counters come back."""
    torch, n = torch_cuda, 1 << 22
    old_k, old_p = po.gen_perm(100_000, 0x5EED1202), po.gen_uniform(100_000, 0x5EED1202, 1, 0, 1 << 20)
    k, p = po.gen_perm(n, 0x5EED1203), po.gen_uniform(n, 0x5EED1203, 1, 0, 1 << 20)
    pk, pp = po.gen_uniform(50021, 0x5EED1204, 0, 0, 200_000), po.gen_uniform(50021, 0x5EED1204, 1, 0, 1 << 20)
    cols, probe_cols, old = [[dev(torch, c) for c in side] for side in ((k, p), (pk, pp), (old_k, old_p))]
    hb = mgv.Op.hash_build(ctx, 0, 1, n)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)
    hb.open(); hb.consume_columns(old, len(old_k)); hb.close()
    hog = leave_free(torch, 16 << 20)
    hb.open()
    with pytest.raises(mgv.MgvError) as e:
        hb.consume_columns(cols, n)
    assert e.value.status == mgv.ENOMEM
    del hog
    torch.cuda.empty_cache()
    rows = {"smaller": 1000, "same": n, "nothing": 0}[then]
    if rows:
        hb.consume_columns(cols, rows)
    hb.close()
    assert hb.result().rows == rows
    probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
    assert agg.result() == po.Chain(k[:rows], p[:rows]).probe_agg(pk, pp)
    for o in (probe, agg, hb):
        o.destroy()


@pytest.mark.parametrize("payloads,lf,share", [(True, 0.5, 0.85), (True, 0.95, 0.93), (False, 0.5, 0.93)])
def test_batch_without_room_for_staging_shares(ctx, torch_cuda, payloads, lf, share):
    """A batch that fits with exact staging ranges only is created and takes them: a histogram and a scan more a run,
    rows that leave their regions (the load factor of 0.95, repeated keys) found by their staging row or key."""
    torch, mix = torch_cuda, []
    for i, (nb, dup) in enumerate([(1 << 23, False), (1_000_003, True), (3000, False), (0, False)]):
        npr = 70_001 + 1000 * i
        cols = make_query_columns(ctx, torch, nb, npr, 1000, 0x5EED1211 + i, dup)
        mix.append(dict(nb=nb, npr=npr, bound=700, G=1000, cols=cols))
    descs = [mgv.query_desc(q["cols"][0], q["nb"], *q["cols"][1:], q["npr"], q["bound"], q["G"],
                            q["cols"][0] if payloads else None) for q in mix]

    def launches(b):
        l0 = ctx.launches
        b.run()
        return ctx.launches - l0

    config = mgv.BatchConfig(lf, 0, 0, 0, 0, 0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    b = mgv.Batch(ctx, descs, config)
    arena = free - torch.cuda.mem_get_info()[0]
    want = launches(b)
    b.destroy()
    hog = leave_free(torch, int(share * arena))
    b = mgv.Batch(ctx, descs, config)
    assert launches(b) == want + 2
    b.run()
    del hog
    torch.cuda.empty_cache()
    for i, q in enumerate(mix):
        assert b.result(i) == oracle_answer(q), i
    b.destroy()


@pytest.mark.parametrize("groups", [1 << 18, 1 << 20])
def test_groupby_without_room_for_sorting(ctx, torch_cuda, groups):
    """A group-by with room for its table and rows but not for sorting space is created; the host orders its rows."""
    torch, n = torch_cuda, 3_000_017
    group = po.gen_uniform(n, 0x5EED1221, 0, -groups // 2, groups)
    value = po.gen_uniform(n, 0x5EED1221, 1, 0, 1 << 20)
    cols = [dev(torch, group), dev(torch, value)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    gb = mgv.Op.groupby(ctx, 0, 1, groups)
    need = free - torch.cuda.mem_get_info()[0]
    gb.destroy()
    hog = leave_free(torch, int(0.8 * need))  # table 20 bytes a slot, rows 24; sorting space 20 to 43
    gb = mgv.Op.groupby(ctx, 0, 1, groups)
    l0 = ctx.launches
    gb.open(); gb.close()
    assert ctx.launches - l0 == 2  # the reset, the packing
    gb.open(); gb.consume_columns(cols, n); gb.close()
    del hog
    torch.cuda.empty_cache()
    g, inverse, count = np.unique(group, return_inverse=True, return_counts=True)
    total = np.zeros(len(g), np.int64)
    np.add.at(total, inverse, value.astype(np.int64))
    assert gb.result() == list(zip(g.tolist(), total.tolist(), count.tolist()))
    gb.destroy()
