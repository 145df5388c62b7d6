"""GPU: index builds as passes over row slots against the oracle and against
the same builds in range CRS (option "row_slots" 0): sizes around the edges of
warps, count groups, conversion blocks and the one-kernel limit, rows of more
runs than a lane's list and of columns wider apart than its mask, and input that
stays in range CRS."""
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


def check(ctx, a, window, slots=True):
    want = orc.dindex(omat(a), *window, algo="hbv")
    da = ctx.upload(a)
    ctx.reset_stats()
    got = ctx.distance_index(da, *window).download()
    st = ctx.stats()
    ctx.set_option("row_slots", 0)
    try:
        ctx.reset_stats()
        crs = ctx.distance_index(da, *window).download()
        crs_st = ctx.stats()
    finally:
        ctx.set_option("row_slots", 1)
    for m in (got, crs):
        assert np.array_equal(m.rowmap, want.rowmap), window
        assert np.array_equal(m.entries, want.entries), window
        assert m.nnz() == want.nnz, window
    # the two forms move different bytes
    if slots is not None:
        assert slots == (st["spgemm_alg_bytes"] != crs_st["spgemm_alg_bytes"])


def rows(a, n):
    """The first n rows and columns of a."""
    rm = a.rowmap[:n + 1]
    e = a.entries[:int(rm[-1])].copy().reshape(-1, 2)
    keep = e[:, 0] < n
    e[:, 1] = np.minimum(e[:, 1], n - 1)
    cnt = np.add.reduceat(np.append(keep, False).astype(np.int64), (rm[:-1] // 2).astype(np.int64)) if n else []
    empty = rm[1:] == rm[:-1]
    cnt = np.where(empty, 0, cnt)
    return CRSMatrix(n, e[keep].reshape(-1), np.concatenate(([0], np.cumsum(2 * cnt))).astype(np.uint64))


GRAPH = None


def graph():
    global GRAPH
    if GRAPH is None:
        GRAPH, _ = gen.graph_adjacency(gen.small_graph_spec(300_000, seed=61))
    return GRAPH


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 65_535, 65_537,
                               131_071, 131_072, 131_073, 131_200, 262_145])
@pytest.mark.parametrize("window", [(3, 11), (0, 70)])
def test_sizes(ctx, n, window):
    check(ctx, rows(graph(), n), window)


@pytest.mark.parametrize("n", [5_000, 140_001])
@pytest.mark.parametrize("window", [(0, 1), (1, 1), (1, 2), (2, 2), (0, 2), (0, 5), (64, 64), (9, 11), (100, 300),
                                    (0, 250), (350, 650), (1000, 1003)])
def test_windows(ctx, n, window):
    check(ctx, rows(graph(), n), window)


@pytest.mark.parametrize("spec", [
    gen.GraphSpec(150_000, 0.02, 0.05, 0.5, 1, 60, 0.0, 0.0, 100, 2000, 5),     # many runs a row
    gen.GraphSpec(150_000, 0.001, 0.004, 0.5, 1, 10, 0.0, 0.5, 100, 4000, 6),   # runs far apart
    gen.GraphSpec(400_000, 0.001, 0.0005, 0.2, 1, 10, 0.0, 0.6, 9000, 20000, 7),  # and past a window
])
@pytest.mark.parametrize("window", [(100, 140), (0, 90), (300, 300)])
def test_branching_graphs(ctx, spec, window):
    a, _ = gen.graph_adjacency(spec)
    check(ctx, a, window)


@pytest.mark.parametrize("hw", [40, 3_000])
@pytest.mark.parametrize("window", [(2, 5), (0, 4)])
def test_columns_anywhere_near(ctx, hw, window):
    # about one short range a row at random in the band: rows fill up quickly
    # (and may fill the arena: the build then falls back)
    a = gen.banded(140_500, hw, 1.2, 1.2, seed=63)
    assert a.entries.size <= 3 * a.numRows() and a.nnz() <= a.entries.size
    check(ctx, a, window, slots=None)


def test_a_full_arena_falls_back(ctx):
    # rows of random columns double with every factor: more ranges than the
    # arena holds, and the build runs again in range CRS
    a = gen.banded(3_000, 3_000, 1.4, 1.0, seed=64)
    want = orc.dindex(omat(a), 12, 12, algo="hbv")
    ctx.reset_stats()
    got = ctx.distance_index(ctx.upload(a), 12, 12).download()
    assert np.array_equal(got.rowmap, want.rowmap) and np.array_equal(got.entries, want.entries)
    assert ctx.stats()["spgemm_reruns"] >= 1


def test_dense_and_noncanonical_input_stays_in_range_crs(ctx):
    check(ctx, gen.random_matrix(2_000, 8_000, seed=65), (1, 3), slots=False)   # 4 ranges a row
    check(ctx, gen.banded(2_000, 200, 1.0, 12.0, seed=66), (1, 3), slots=False)  # ranges of 12 columns
    split = CRSMatrix(6, np.array([1, 1, 2, 3, 3, 3, 5, 5], np.uint32), np.array([0, 4, 6, 6, 8, 8, 8], np.uint64))
    check(ctx, split, (1, 3), slots=False)


@pytest.mark.parametrize("n", [33, 131_073])
@pytest.mark.parametrize("k", [0, 1, 2, 3, 63, 64, 100])
def test_powers(ctx, n, k):
    a = rows(graph(), n)
    want = orc.power(omat(a), k, algo="hbv")
    got = ctx.power(ctx.upload(a), k).download()
    assert np.array_equal(got.rowmap, want.rowmap) and np.array_equal(got.entries, want.entries)
    assert got.nnz() == want.nnz


def test_a_batch_of_chains_beside_range_crs_builds(ctx):
    # parts of a chain around the edges of its blocks, several windows side by
    # side, graphs that stay in range CRS, and one whose chain runs full
    windows = [(100, 300), (0, 50), (3, 3), (1, 1), (0, 1), (200, 500)]
    graphs = [rows(graph(), n) for n in (1, 50, 1023, 1024, 1025, 2048, 3000, 20_000, 70_001, 1024, 31, 4096)]
    ws = [windows[k % len(windows)] for k in range(len(graphs))]
    graphs += [gen.random_matrix(500, 2_500, seed=67), gen.banded(3_000, 3_000, 1.4, 1.0, seed=64),
               CRSMatrix(0, np.zeros(0, np.uint32), np.zeros(1, np.uint64))]
    ws += [(1, 3), (12, 12), (1, 3)]
    for _ in range(2):
        ctx.reset_stats()
        got = ctx.batch_distance_index([ctx.upload(g) for g in graphs], ws)
        assert ctx.stats()["graph_launches"] == 1
        for k, (g, w) in enumerate(zip(graphs, ws)):
            want = orc.dindex(omat(g), *w, algo="hbv")
            m = got[k].download()
            assert np.array_equal(m.rowmap, want.rowmap) and np.array_equal(m.entries, want.entries), (k, w)
            assert m.nnz() == want.nnz, (k, w)


def product_forms(n, seed):
    """Factors that single products take in slots, and their neighbours that they
    do not: a row of several short ranges, rows split or out of order, ranges of
    12 columns, a wide matrix."""
    a = rows(graph(), n)
    yield "square", a, a, True
    yield "another factor", a, gen.banded(n, 50, 1.2, 1.2, seed=seed), True
    yield "and before it", gen.banded(n, 50, 1.2, 1.2, seed=seed), a, True
    yield "dense left", gen.random_matrix(n, 3 * n, seed=seed + 1), a, False
    yield "dense right", a, gen.banded(n, 200, 1.0, 12.0, seed=seed + 2), False
    i = np.arange(n - 1, dtype=np.uint32)  # [i, i], and in every third row [i + 1, i + 1] beside it
    both = np.stack([i, i, i + 1, i + 1], 1)
    entries = both[np.repeat((i % 3 == 0)[:, None], 4, 1) | np.array([True, True, False, False])]
    at = np.concatenate(([0], np.cumsum(np.where(i % 3 == 0, 4, 2)))).astype(np.uint64)
    yield "split rows", CRSMatrix(n, entries, np.append(at, at[-1])), a, False


@pytest.mark.parametrize("n", [24_575, 24_576, 24_577, 33_023, 131_072, 131_073])
def test_single_products(ctx, n):
    for what, a, b, slots in product_forms(n, 71):
        da = ctx.upload(a)
        db = da if b is a else ctx.upload(b)
        want = orc.spgemm(omat(a), omat(b))
        ctx.reset_stats()
        got = ctx.spgemm(da, db).download()
        here = ctx.stats()["kernel_launches"]
        ctx.set_option("row_slots", 0)
        try:
            ctx.reset_stats()
            crs = ctx.spgemm(da, db).download()
            there = ctx.stats()["kernel_launches"]
        finally:
            ctx.set_option("row_slots", 1)
        for m in (got, crs):
            assert np.array_equal(m.rowmap, want.rowmap), what
            assert np.array_equal(m.entries, want.entries), what
            assert m.nnz() == want.nnz, what
        assert (here != there) == (slots and n >= 24_576), what


def test_results_past_the_early_room(ctx):
    # more than two ranges a row: the result is written again once its size is known
    a = gen.banded(30_000, 3_000, 1.48, 1.0, seed=72)
    da = ctx.upload(a)
    assert a.entries.size <= 3 * a.numRows() and a.nnz() <= a.entries.size
    for _ in range(2):
        ctx.reset_stats()
        got = ctx.power(da, 2).download()
        want = orc.power(omat(a), 2, algo="hbv")
        assert got.entries.size > 4 * a.numRows()
        assert np.array_equal(got.rowmap, want.rowmap) and np.array_equal(got.entries, want.entries)
        assert got.nnz() == want.nnz and ctx.stats()["spgemm_reruns"] == 0
