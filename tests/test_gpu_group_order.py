"""Groups ordered on the device: result sizes on both sides of every change of
method (host order, counting, one CTA in shared memory, one CTA in global
memory, more rows than the landing zone), dense, sparse and extreme groups, and
a table reopened after each close."""
import numpy as np
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


def groups_of(kind, distinct, rows, seed):
    """`rows` group values, `distinct` of them different."""
    ids = np.arange(distinct, dtype=np.int64)
    if kind == "dense":
        vals = ids
    elif kind == "sparse":  # an odd multiplier permutes the 32-bit integers
        vals = (ids * 2654435761 + 12345) % (1 << 32)
    else:  # both ends of the range and around zero
        vals = np.where(ids % 2 == 0, -(1 << 31) + ids // 2, (1 << 31) - 1 - ids // 2)
    vals = vals.astype(np.uint32).view(np.int32) if kind == "sparse" else vals.astype(np.int32)
    pick = po.gen_uniform(rows, seed, 0, 0, distinct)
    pick[:distinct] = np.arange(distinct)  # every value occurs
    return vals[pick]


def want_rows(group, value):
    g, inverse, count = np.unique(group, return_inverse=True, return_counts=True)
    total = np.zeros(len(g), np.int64)
    np.add.at(total, inverse, value.astype(np.int64))
    return [(int(a), int(b), int(c)) for a, b, c in zip(g, total, count)]


@pytest.mark.parametrize("kind", ["dense", "sparse", "extreme"])
@pytest.mark.parametrize("distinct", [1, 64, 65, 511, 513, 1025, 4096, 4097, 8191, 8200, 32769, 70001])
def test_groupby_order(ctx, torch_cuda, distinct, kind):
    gb = mgv.Op.groupby(ctx, 0, 1, distinct)
    for turn in range(3):  # the second and third open find the table as the close before left it
        d = max(1, distinct >> turn)
        rows = 2 * d + 37
        group = groups_of(kind, d, rows, 0x5EED0D01 + turn)
        value = po.gen_uniform(rows, 0x5EED0D01 + turn, 1, -(1 << 31), 1 << 32)
        gb.open(); gb.consume_columns([dev(torch_cuda, group), dev(torch_cuda, value)], rows); gb.close()
        assert gb.result() == want_rows(group, value)
    gb.open(); gb.close()
    assert gb.result() == []
    gb.destroy()


@pytest.mark.parametrize("kind", ["dense", "sparse"])
def test_batch_order(ctx, torch_cuda, kind):
    """Queries of one batch with 1 to 40000 groups, more groups than fit shared
    memory among them, in group order after every run."""
    queries, want, keep = [], [], []
    for i, distinct in enumerate([1, 500, 600, 8193, 8194, 40000]):
        rows = 2 * distinct + 11
        group = groups_of(kind, distinct, rows, 0x5EED0D11 + i)
        value = po.gen_uniform(rows, 0x5EED0D11 + i, 1, 0, 1 << 20)
        key = (np.arange(rows) % 7).astype(np.int32)  # every row joins once
        cols = [dev(torch_cuda, c) for c in (np.arange(7, dtype=np.int32), key, np.zeros(rows, np.int32), group, value)]
        keep.append(cols)
        queries.append(mgv.query_desc(cols[0], 7, cols[1], cols[2], cols[3], cols[4], rows, 0, distinct))
        want.append(want_rows(group, value))
    b = mgv.Batch(ctx, queries, mgv.BatchConfig(0.5, 0, 0, 0, 1, 0), keep)
    for _ in range(3):  # launched, captured, replayed
        b.run()
        assert [b.result(q) for q in range(len(queries))] == want
    b.run_plain()
    assert [b.result(q, plain=True) for q in range(len(queries))] == want
    b.destroy()
