"""One batch's results read by several threads at once."""
from concurrent.futures import ThreadPoolExecutor

import pytest

import mgv
from querymix import make_mix, oracle_answer

pytestmark = pytest.mark.gpu


def test_results_read_by_many_threads(ctx, torch_cuda):
    """Queries of up to 64 groups, whose rows the host orders, and larger ones, ordered by the device: every reader
    gets every query's rows, from the batch and from the plain pipeline, after every run."""
    mix = make_mix(ctx, torch_cuda, 24, 17, groups=(2, 8))
    want = [oracle_answer(q) for q in mix]
    assert any(q["G"] <= 64 for q in mix) and any(q["G"] > 64 for q in mix)
    b = mgv.Batch(ctx, [mgv.query_desc(q["cols"][0], q["nb"], *q["cols"][1:], q["npr"], q["bound"], q["G"])
                        for q in mix])

    def read(_):
        return [[b.result(i, plain) for i in range(len(mix))] for plain in (True, False)]

    with ThreadPoolExecutor(8) as pool:
        for _ in range(5):
            b.run()
            b.run_plain()
            for got in pool.map(read, range(16)):
                assert got == [want, want]
    b.destroy()
