"""Probe -> aggregate over column slices that start at any row: keys and
payloads each 0 to 3 rows past a 16-byte boundary, row counts around whole
tiles of the staged probe (1024 or 2048 rows), and operators opened again
after every close (whose sums start from zero without a clearing call)."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,rows_per_thread", [(3, 4), (2, 4), (3, 8)])
@pytest.mark.parametrize("payload", [True, False])
@pytest.mark.parametrize("dups", [True, False])
def test_probe_of_slices(ctx, torch_cuda, dups, payload, kernel, rows_per_thread):
    nb = 5000
    bk = po.gen_uniform(nb, 0x5EED1001, 0, 0, 1500) if dups else po.gen_perm(nb, 0x5EED1001)
    bp = po.gen_uniform(nb, 0x5EED1001, 1, -(1 << 31), 1 << 32)
    pk = po.gen_uniform(300 * 1024, 0x5EED1002, 0, 0, 6000)
    pk[::97] = -(1 << 31)
    pp = po.gen_uniform(len(pk), 0x5EED1002, 1, -(1 << 31), 1 << 32)
    dk, dp = dev(torch_cuda, pk), dev(torch_cuda, pp)
    chain = po.Chain(bk, bp)
    old = ctx.tuning()
    ctx.set_tuning(probe_kernel=kernel, probe_rows_per_thread=rows_per_thread)
    hb = mgv.Op.hash_build(ctx, 0, 1, nb)
    agg = mgv.Op.aggregate(ctx, 1 if payload else -1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)
    try:
        hb.open(); hb.consume_columns([dev(torch_cuda, bk), dev(torch_cuda, bp)], nb); hb.close()
        for k0 in range(4):
            for p0 in range(4):
                for n in (1, 3, 7, 8, 1023, 1024, 1031, 1032, 2049, 2055, 3072, 250001):
                    k, p = pk[k0:k0 + n], pp[p0:p0 + n]
                    probe.open(); probe.consume_columns([dk[k0:], dp[p0:]], n); probe.close()
                    want = chain.probe_agg(k, p if payload else np.zeros(n, np.int32))
                    assert agg.result() == want, (k0, p0, n)
        probe.open(); probe.close()
        assert agg.result() == (0, 0)
    finally:
        ctx.set_tuning(probe_kernel=old.probe_kernel, probe_rows_per_thread=old.probe_rows_per_thread)
        for o in (probe, agg, hb):
            o.destroy()
