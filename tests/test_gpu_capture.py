"""Operators whose open and consume were captured into a CUDA graph, replayed
before and after a close, and then opened, fed and closed in the ordinary way:
an open starts from nothing whatever a replay left on the device."""
import pytest

import mgv
import pyoracle as po
from gpu_util import dev

pytestmark = pytest.mark.gpu


def capture(torch, head, cols, n):
    """A graph of one open and one consume on a stream of its own; the operator is left open."""
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        head.open(stream=st.cuda_stream)
        head.consume_columns(cols, n, stream=st.cuda_stream)

    def replay():
        with torch.cuda.stream(st):
            g.replay()

    return st, replay


def result_chains(ctx, torch, n):
    """name -> (head, its columns, terminal, other columns): select -> aggregate, probe -> aggregate, select ->
    group-by of tables closed by one CTA and by many."""
    nb = 3000
    hb = mgv.Op.hash_build(ctx, 0, 1, nb)
    bk, bp = po.gen_perm(nb, 0x5EED1101), po.gen_uniform(nb, 0x5EED1101, 1, 0, 1 << 20)
    hb.open(); hb.consume_columns([dev(torch, bk), dev(torch, bp)], nb); hb.close()
    agg, pagg = mgv.Op.aggregate(ctx, 0, -1), mgv.Op.aggregate(ctx, 1, 2)
    small, large = mgv.Op.groupby(ctx, 0, 1, 1000), mgv.Op.groupby(ctx, 0, 1, 5000)
    heads = {"select_agg": (mgv.Op.select(ctx, 1, 499, agg), agg),
             "probe_agg": (mgv.Op.hash_probe(ctx, 0, hb, pagg), pagg),
             "group_small": (mgv.Op.select(ctx, 1, 499, small), small),
             "group_large": (mgv.Op.select(ctx, 1, 499, large), large)}
    sides = [[po.gen_uniform(n, 0x5EED1102 + i, 0, 0, 1000), po.gen_uniform(n, 0x5EED1102 + i, 1, 0, 1000)]
             for i in range(2)]
    return heads, [[dev(torch, c) for c in s] for s in sides], hb


@pytest.mark.parametrize("chain", ["select_agg", "probe_agg", "group_small", "group_large"])
@pytest.mark.parametrize("open_captured", [True, False])
def test_plain_pass_after_a_replay(ctx, torch_cuda, chain, open_captured):
    torch, n = torch_cuda, 60_007
    heads, sides, hb = result_chains(ctx, torch, n)
    head, term = heads[chain]

    def plain(i):
        head.open(); head.consume_columns(sides[i], n); head.close()
        return term.result()

    want = [plain(0), plain(1)]
    assert want[0] != want[1]
    if open_captured:
        st, replay = capture(torch, head, sides[1], n)
    else:  # the consume alone
        head.open()
        st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=st):
            head.consume_columns(sides[1], n, stream=st.cuda_stream)

        def replay():
            with torch.cuda.stream(st):
                g.replay()
    replay()
    head.close(stream=st.cuda_stream)
    assert term.result() == want[1]
    replay()
    torch.cuda.synchronize()
    assert plain(0) == want[0]
    replay()
    replay()
    torch.cuda.synchronize()
    assert plain(1) == want[1]
    assert plain(0) == want[0]
    head.open(); head.close()
    assert term.result() in ((0, 0), [])
    for h, t in heads.values():
        h.destroy(); t.destroy()
    hb.destroy()


@pytest.mark.parametrize("radix_bits", [0, 4])
@pytest.mark.parametrize("captured_rows,plain_rows", [(30_000, 150_001), (150_001, 30_000), (3_000, 150_001)])
def test_replayed_build_is_closed_by_its_own_counters(ctx, torch_cuda, captured_rows, plain_rows, radix_bits):
    """A graph of one build replayed over the rows of another, by any of the build paths: the close reads the
    counters of the table as it is, whichever of them wrote it last."""
    torch = torch_cuda
    pk, pp = po.gen_uniform(20011, 0x5EED1112, 0, 0, 1 << 17), po.gen_uniform(20011, 0x5EED1112, 1, 0, 1 << 20)
    probe_cols = [dev(torch, pk), dev(torch, pp)]
    sides = []
    for i, n in enumerate((captured_rows, plain_rows)):
        keys = po.gen_perm(n, 0x5EED1113 + i) if i else po.gen_uniform(n, 0x5EED1113, 0, 0, n // 2)  # captured: repeated
        sides.append((keys, po.gen_uniform(n, 0x5EED1113 + i, 1, 0, 1 << 20)))
    cols = [[dev(torch, c) for c in side] for side in sides]
    hb = mgv.Op.hash_build(ctx, 0, 1, max(captured_rows, plain_rows), radix_bits=radix_bits)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)

    def check(i):
        assert hb.result().rows == len(sides[i][0])
        assert hb.result().has_duplicates == (1 - i)
        probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
        assert agg.result() == po.Chain(*sides[i]).probe_agg(pk, pp)

    def build(i):
        hb.open(); hb.consume_columns(cols[i], len(sides[i][0])); hb.close()
        check(i)

    build(0)
    build(1)
    st, replay = capture(torch, hb, cols[0], captured_rows)
    replay()
    hb.close(stream=st.cuda_stream)
    check(0)
    hb.open(); hb.consume_columns(cols[1], plain_rows)
    torch.cuda.synchronize()
    replay()
    hb.close(stream=st.cuda_stream)
    check(0)
    build(1)
    for o in (probe, agg, hb):
        o.destroy()


@pytest.mark.parametrize("rows", [1000, 30_000, 150_001])
def test_build_by_a_replay_alone(ctx, torch_cuda, rows):
    """Open, replay of a captured build, close: the table holds the replay's rows.  Open, close: it is empty."""
    torch, room = torch_cuda, 150_001
    side = po.gen_perm(rows, 0x5EED1121), po.gen_uniform(rows, 0x5EED1121, 1, 0, 1 << 20)
    other = po.gen_perm(room, 0x5EED1122), po.gen_uniform(room, 0x5EED1122, 1, 0, 1 << 20)
    pk, pp = po.gen_uniform(20011, 0x5EED1123, 0, 0, 1 << 17), po.gen_uniform(20011, 0x5EED1123, 1, 0, 1 << 20)
    cols, other_cols, probe_cols = [[dev(torch, c) for c in s] for s in (side, other, (pk, pp))]
    none = [c[:0] for c in side]
    hb = mgv.Op.hash_build(ctx, 0, 1, room)
    agg = mgv.Op.aggregate(ctx, 1, 2)
    probe = mgv.Op.hash_probe(ctx, 0, hb, agg)

    def check(s):
        assert hb.result().rows == len(s[0])
        probe.open(); probe.consume_columns(probe_cols, len(pk)); probe.close()
        assert agg.result() == po.Chain(*s).probe_agg(pk, pp)

    def build(s, c):
        hb.open(); hb.consume_columns(c, len(s[0])); hb.close()
        check(s)

    build(side, cols)
    build(other, other_cols)
    st, replay = capture(torch, hb, cols, rows)
    replay()
    hb.close(stream=st.cuda_stream)
    check(side)
    for _ in range(2):
        build(other, other_cols)
        hb.open(stream=st.cuda_stream)
        replay()
        hb.close(stream=st.cuda_stream)
        check(side)
        hb.open(); hb.close()
        check(none)
    for o in (probe, agg, hb):
        o.destroy()
