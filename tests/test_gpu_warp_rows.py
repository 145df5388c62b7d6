"""GPU: rows of a row-slot chain that a warp walks, against the oracle: spans around
the reach of a row's bitmaps, numbers of runs and of columns around a lane's limits,
more such rows than the queue holds, and what such rows cost."""
import time

import numpy as np
import pytest

from diverg_b200 import CRSMatrix, gen
from diverg_b200.runtime import Context
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def omat(m):
    return orc.OMat(m.numRows(), m.numCols(), m.rowmap, m.entries, m.nnz())


def path_and(n, extra):
    """The path i -> i + 1 with rows of `extra` {row: [(first, last), ...]}, canonical."""
    rows = [[(i + 1, i + 1)] if i + 1 < n else [] for i in range(n)]
    for r, ranges in extra.items():
        rows[r] = sorted(ranges)
    rm = np.concatenate(([0], np.cumsum([2 * len(r) for r in rows]))).astype(np.uint64)
    return CRSMatrix(n, np.array([c for r in rows for v in r for c in v], np.uint32), rm)


def check(ctx, a, window):
    want = orc.dindex(omat(a), *window, algo="hbv")
    d = ctx.upload(a)
    ctx.reset_stats()
    got = ctx.distance_index(d, *window).download()
    assert np.array_equal(got.rowmap, want.rowmap), window
    assert np.array_equal(got.entries, want.entries), window
    assert got.nnz() == want.nnz, window
    return ctx.stats()


@pytest.mark.parametrize("n", [40_000, 140_000])  # both forms of a pass
@pytest.mark.parametrize("window", [(0, 6), (5, 5), (3, 30)])
def test_runs_columns_and_spans(ctx, n, window):
    extra, at = {}, 100
    # singles `step` apart: 7 to 10 runs, and spans around the bitmaps' words
    for runs in (7, 8, 9, 10, 40):
        for span in (30, 1000, 8150, 10_200, 10_239, 10_240, 10_241, 12_300, 20_000):
            step = max(2, span // runs)
            extra[at] = [(at + 1, at + 1)] + [(at + 1 + step * k, at + 1 + step * k) for k in range(1, runs)]
            at += 41
    # ranges of 1 to 1000 columns, one and several
    for length in (2, 63, 64, 65, 255, 256, 257, 300, 1000):
        extra[at] = [(at + 1, at + length)]
        extra[at + 40] = [(at + 41, at + 41), (at + 45, at + 44 + length), (at + 2500, at + 2499 + length // 2 + 1)]
        at += 83
    # a lower column than the row's others, before and within the bitmaps' margin
    for back in (30, 1900, 2100, 3000):
        extra[at] = [(at - back, at - back)] + [(at + 3 * k, at + 3 * k) for k in range(1, 12)]
        at += 3100
    assert at + 20_001 < n
    check(ctx, path_and(n, extra), window)


@pytest.mark.parametrize("n", [40_000, 140_000])
def test_more_rows_than_the_queue_holds(ctx, n):
    # every row of a long stretch has 12 runs; chains that fit their arena
    a = path_and(n, {r: [(r + 1 + 5 * k, r + 1 + 5 * k) for k in range(12)] for r in range(500, 500 + n // 30)})
    st = check(ctx, a, (2, 2))
    assert st["spgemm_reruns"] == 0 and st["spgemm_slow_rows"] >= n // 30
    b = path_and(n, {r: [(r + 1 + 5 * k, r + 1 + 5 * k) for k in range(4)] for r in range(500, 500 + n // 4)})
    st = check(ctx, b, (2, 4))
    assert st["spgemm_reruns"] == 0 and st["spgemm_slow_rows"] > max(1024, n // 8)


def test_rows_of_many_runs_cost_no_more_than_in_range_crs(ctx):
    # A^300 of a variant-dense graph: 2 ranges a row on average, and 4,000 rows of
    # more runs than a lane's list in clumps
    a, _ = gen.graph_adjacency(gen.small_graph_spec(1_000_000, seed=3))
    d = ctx.upload(a)
    took, forms = {}, []
    for slots in (1, 0):
        ctx.set_option("row_slots", slots)
        try:
            ctx.reset_stats()
            m = ctx.power(d, 300)
            if slots:
                st = ctx.stats()
                assert st["spgemm_reruns"] == 0 and st["spgemm_slow_rows"] >= 1000
            forms.append(m.download())
            m.free()
            best = 1e9
            for _ in range(5):
                t = time.perf_counter()
                ctx.power(d, 300).free()
                best = min(best, time.perf_counter() - t)
            took[slots] = best
        finally:
            ctx.set_option("row_slots", 1)
    assert np.array_equal(forms[0].rowmap, forms[1].rowmap) and np.array_equal(forms[0].entries, forms[1].entries)
    assert took[1] <= 1.5 * took[0], took
