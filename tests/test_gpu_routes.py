"""GPU: which way a call takes, and what it holds on to: matrices whose caller gave
another column count than the true one, results' memory, chains that do not fit."""
import time

import numpy as np
import pytest

from diverg_b200 import CRSMatrix, gen
from diverg_b200.runtime import Context
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    c = Context(0)
    yield c
    c.close()


def omat(m):
    return orc.OMat(m.numRows(), m.numCols(), m.rowmap, m.entries, m.nnz())


def same(got, want, what):
    assert np.array_equal(got.rowmap, want.rowmap), what
    assert np.array_equal(got.entries, want.entries), what
    assert got.nnz() == want.nnz, what


def wrapped(ctx, m, nnz):
    """m's arrays on the device, and the matrix that wraps them."""
    import torch
    t = [torch.from_numpy(x.view(d).copy()).cuda() for x, d in ((m.rowmap, np.int64), (m.entries, np.int32))]
    return t, ctx.wrap_device(m.numRows(), m.numCols(), t[0].data_ptr(), t[1].data_ptr(), m.entries.size, nnz)


def inputs():
    n = 30_000
    yield "graph", gen.graph_adjacency(gen.small_graph_spec(n, seed=81))[0], (100, 300)
    yield "ranges of 6", gen.banded(n, 200, 1.0, 6.0, seed=82), (1, 3)
    yield "ranges of 40", gen.banded(n, 200, 1.0, 40.0, seed=83), (1, 2)


@pytest.mark.parametrize("form", ["wrap", "upload", "upload_u32"])
def test_a_wrong_column_count_changes_no_route(form):
    for what, m, window in inputs():
        true, seen = m.nnz(), []
        for nnz in (true, 1, 10 ** 9) + ((0,) if form == "wrap" else ()):
            ctx, keep = Context(0), None  # (a context's estimates follow its earlier calls)
            if form == "wrap":
                keep, d = wrapped(ctx, m, nnz)
            else:
                rm = m.rowmap.astype(np.uint32) if form == "upload_u32" else m.rowmap
                u = CRSMatrix(m.numCols(), m.entries, rm, nnz, size_type=rm.dtype.type)
                d = ctx.upload(u)
            assert d.nnz == nnz, what  # what the caller said is what the caller is told
            route = []
            for call in (lambda: ctx.spgemm(d, d), lambda: ctx.power(d, 3), lambda: ctx.distance_index(d, *window)):
                ctx.reset_stats()
                r = call()
                st = ctx.stats()
                route.append((st["spgemm_alg_bytes"], st["spgemm_light"], st["spgemm_levels"]))
                got = r.download()
                r.free()
            seen.append((nnz, route))
            if nnz != true:
                same(got, orc.dindex(omat(m), *window, algo="hbv"), what)
            d.free()
            ctx.close()
            del keep
        assert all(route == seen[0][1] for _, route in seen), (what, seen)


def used_bytes(ctx):
    """Device memory in use from CUDA's pool (what contexts allocate from), their caches given back."""
    from cuda.bindings import runtime as rt
    ctx.trim()
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert int(err) == 0
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert int(err) == 0
    return int(used)


def block(nbytes):
    """The size of the block that holds nbytes (the allocator's classes)."""
    nbytes = (nbytes + 255) // 256 * 256
    if nbytes <= 1 << 20:
        return nbytes
    step = 1 << (nbytes.bit_length() - 3)
    return (nbytes + step - 1) // step * step


@pytest.mark.parametrize("bases,window", [(3_000_000, (400, 600)), (3_000_000, (7, 9)), (40_000, (100, 300))])
def test_an_index_holds_no_more_than_it_needs(ctx, bases, window):
    # at most a quarter and 1 MiB more than its entries, whichever route built it
    a, _ = gen.graph_adjacency(gen.chromosome_graph_spec(bases, seed=84))
    d = ctx.upload(a)
    for slots in (1, 0, 1):
        ctx.set_option("row_slots", slots)
        ctx.distance_index(d, *window).free()
        before = used_bytes(ctx)
        m = ctx.distance_index(d, *window)
        held = used_bytes(ctx) - before
        # (a cached block of up to a quarter more may serve the entries)
        most = block(8 * (m.nrows + 1) + 16) + 5 * block(5 * m.nentries + (1 << 20) + 16) // 4
        assert held <= most, (slots, held, most)
        m.free()


def path_and(n, extra):
    """The path i -> i + 1, with the ranges `extra` in place of the rows that it names."""
    i = np.arange(n - 1, dtype=np.uint32)
    rows = np.split(np.stack([i + 1, i + 1], 1), range(1, n - 1)) + [np.zeros((0, 2), np.uint32)]
    for r, e in extra.items():
        rows[r] = np.asarray(e, np.uint32).reshape(-1, 2)
    rm = np.concatenate(([0], np.cumsum([2 * len(r) for r in rows]))).astype(np.uint64)
    return CRSMatrix(n, np.concatenate(rows).reshape(-1), rm)


def index(ctx, d, m, window):
    """The index, held against the oracle, and how often its products ran again."""
    ctx.reset_stats()
    r = ctx.distance_index(d, *window)
    again = ctx.stats()["spgemm_reruns"]
    same(r.download(), orc.dindex(omat(m), *window, algo="hbv"), window)
    r.free()
    return again


def test_chains_that_do_not_fit_are_not_tried_on_every_call(ctx):
    # rows of random columns double with every factor, past any arena
    m = gen.banded(30_000, 30_000, 1.0, 1.0, seed=85)
    d = ctx.upload(m)
    ctx.set_option("row_slots", 0)
    crs = min(index(ctx, d, m, (8, 9)) for _ in range(3))
    ctx.set_option("row_slots", 1)
    again = [index(ctx, d, m, (8, 9)) - crs for _ in range(16)]
    # a larger arena, then 1, 3, 7 calls between two attempts
    assert 1 <= sum(a > 0 for a in again) <= 5, again
    # a matrix of another kind is tried
    g, _ = gen.graph_adjacency(gen.small_graph_spec(30_000, seed=86))
    assert index(ctx, ctx.upload(g), g, (8, 9)) == 0


def test_batches_with_a_graph_that_does_not_fit(ctx):
    m = gen.banded(30_000, 30_000, 1.0, 1.0, seed=85)
    g, _ = gen.graph_adjacency(gen.small_graph_spec(20_000, seed=87))
    graphs = [m, g, g, m]
    wants = [orc.dindex(omat(x), 8, 9, algo="hbv") for x in graphs]
    up = [ctx.upload(x) for x in graphs]
    for _ in range(6):
        for got, want in zip(ctx.batch_distance_index(up, [(8, 9)] * 4), wants):
            same(got.download(), want, "batch")
            got.free()


def test_rows_that_reach_far_are_left_to_range_crs(ctx):
    n = 200_000
    m = path_and(n, {777: [[778, 20_777]]})
    d = ctx.upload(m)
    assert index(ctx, d, m, (40, 60)) >= 1
    assert index(ctx, d, m, (40, 60)) == 0  # (and not tried at once again)
    # a few that reach past the bitmaps, and name few columns, stay
    m = path_and(n, {r: [[r + 1 + 1900 * k, r + 1 + 1900 * k] for k in range(12)] for r in (500, 600, 90_000)})
    assert index(ctx, ctx.upload(m), m, (3, 5)) == 0


def peak_bytes(ctx, call):
    """The most device memory in use from CUDA's pool during a call."""
    from cuda.bindings import driver, runtime as rt
    before = used_bytes(ctx)
    _, pool = rt.cudaDeviceGetDefaultMemPool(0)
    high = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    err, = rt.cudaMemPoolSetAttribute(pool, high, driver.cuuint64_t(0))
    assert int(err) == 0
    call()
    err, most = rt.cudaMemPoolGetAttribute(pool, high)
    assert int(err) == 0
    return int(most) - before


def test_a_row_of_too_many_ranges_makes_no_arena_larger(ctx):
    n = 200_000
    g = path_and(n, {5: [[6, 6], [9, 9]]})
    d = ctx.upload(g)
    build = lambda: ctx.distance_index(d, 20, 30).free()
    build()
    usual = peak_bytes(ctx, build)
    many = path_and(n, {100: [[101 + 2 * k, 101 + 2 * k] for k in range(70_000)]})  # past 65,534
    assert index(ctx, ctx.upload(many), many, (1, 1)) >= 1
    assert peak_bytes(ctx, build) <= usual * 1.02


@pytest.mark.parametrize("n,dense_slots", [(1 << 18, True), ((1 << 18) + 1, False), (400_000, False)])
def test_large_dense_input_stays_in_range_crs(ctx, n, dense_slots):
    # more than a quarter of a column a row beyond its first, of the rows that have any
    g, _ = gen.graph_adjacency(gen.small_graph_spec(n - 8_000, seed=88))
    for what, m, slots in (("graph", g, True), ("1.4 a row", gen.banded(n, 40, 1.2, 1.2, seed=89), dense_slots),
                           ("0.9 a row", gen.banded(n, 40, 0.9, 1.0, seed=90), dense_slots)):
        assert m.entries.size <= 3 * m.numRows() and m.nnz() <= m.entries.size, what
        d = ctx.upload(m)
        for call in (lambda: ctx.spgemm(d, d), lambda: ctx.power(d, 2), lambda: ctx.distance_index(d, 1, 2)):
            ctx.set_option("row_slots", 0)
            call().free()  # (builds in range CRS size themselves by the one before)
            moved, forms = [], []
            for on in (1, 0):
                ctx.set_option("row_slots", on)
                ctx.reset_stats()
                r = call()
                moved.append(ctx.stats()["spgemm_alg_bytes"])
                forms.append(r.download())
                r.free()
            ctx.set_option("row_slots", 1)
            assert np.array_equal(forms[0].rowmap, forms[1].rowmap), what
            assert np.array_equal(forms[0].entries, forms[1].entries), what
            assert (moved[0] != moved[1]) == slots, (what, moved)
        d.free()


def test_an_adjacency_matrix_holds_no_more_than_it_needs(ctx):
    # one range a row, however many edges in a row make it
    n = 2_000
    u = np.repeat(np.arange(1, n, dtype=np.uint32), np.arange(n - 1, 0, -1))
    v = np.concatenate([np.arange(k + 1, n + 1, dtype=np.uint32) for k in range(1, n)])
    for lower, upper in ((1, 0), (1, n), (5, n + 1)):
        before = used_bytes(ctx)
        edges = np.stack([u, v], 1)
        if upper == n:
            edges = edges[v < n]  # (none leaves the node range)
        m = ctx.adjacency_from_graph(np.ones(n, np.uint32), edges, lower, upper)
        held = used_bytes(ctx) - before
        assert held <= block(8 * (m.nrows + 1) + 16) + 5 * block(5 * m.nentries + (1 << 20) + 16) // 4, held
        rows = (upper or n + 1) - lower
        assert m.nentries == 2 * (rows - 1) and m.nnz == rows * (rows - 1) // 2
        m.free()


def cycle(n, steps):
    """Row i holds the columns i + s modulo n for the steps s."""
    cols = np.sort((np.arange(n)[:, None] + np.array(steps)) % n, axis=1)
    rows = [[(c[0], c[0])] for c in cols] if len(steps) == 1 else None
    if rows is None:
        rows = []
        for c in cols:
            r = []
            for x in c:
                if r and r[-1][1] + 1 == x:
                    r[-1] = (r[-1][0], x)
                else:
                    r.append((x, x))
            rows.append(r)
    rm = np.concatenate(([0], np.cumsum([2 * len(r) for r in rows]))).astype(np.uint64)
    return CRSMatrix(n, np.array([x for r in rows for v in r for x in v], np.uint32), rm)


@pytest.mark.parametrize("window", [(2 ** 31 + 5, 2 ** 31 + 5), (3_000_000_000, 3_000_000_002), (2 ** 32 - 1, 2 ** 32 - 1)])
def test_large_exponents_are_planned_at_once(ctx, window):
    # a chain over a cycle takes some 40 passes, whatever the exponent
    m = cycle(1_000, (1,))
    d = ctx.upload(m)
    want = orc.dindex(omat(m), *window, algo="hbv")
    ctx.distance_index(d, 5, 9).free()
    t = time.perf_counter()
    r = ctx.distance_index(d, *window)
    took = time.perf_counter() - t
    same(r.download(), want, window)
    assert took < 0.3, took


@pytest.mark.parametrize("window", [(0, 2 ** 32 - 1), (2 ** 32 - 1, 2 ** 32 - 1), (2 ** 31 + 1, 2 ** 32 - 1), (7, 2 ** 31)])
def test_large_exponents_where_a_pass_takes_one_factor(ctx, window):
    # two columns a row: A^dmin by factors of A alone would take up to 2^32 - 1 passes
    m = cycle(300, (1, 2))
    d = ctx.upload(m)
    t = time.perf_counter()
    r = ctx.distance_index(d, *window)
    took = time.perf_counter() - t
    same(r.download(), orc.dindex(omat(m), *window, algo="hbv"), window)
    assert took < 1.0, took


@pytest.mark.parametrize("window", [(0, 1), (1, 1), (0, 2), (3, 5), (0, 250), (400, 600)])
def test_the_server_reserves_what_a_build_takes(window):
    # a budget below what a build of 4e6 bases takes admits none, even with the largest arena
    from diverg_b200.serving import Server
    a, _ = gen.graph_adjacency(gen.chromosome_graph_spec(4_000_000, seed=93))
    held = 8 * (a.numRows() + 1) + 4 * a.entries.size
    ctx = Context(0)
    dense = gen.banded(3_000, 3_000, 1.4, 1.0, seed=64)  # (fills its arena: the next one is larger)
    dd = ctx.upload(dense)
    ctx.distance_index(dd, 12, 12).free()
    d = ctx.upload(a)
    took = held + peak_bytes(ctx, lambda: ctx.batch_distance_index([d], [window])[0].free())
    d.free()
    ctx.close()
    with Server(hbm_budget_bytes=took - 1) as s:
        req = s.submit_build(a, *window)
        assert s.wait([req])[0]["status"] != 0


@pytest.mark.parametrize("n", [1, 300, 5_000])
@pytest.mark.parametrize("ranges,single", [(400, True), (455, True), (456, False), (600, False)])
def test_sums_of_dense_rows(ctx, n, ranges, single):
    # up to 910 ranges a row of both operands together in one pass (one launch), denser
    # rows in two
    ncols = 4 * ranges + 8
    rng = np.random.default_rng(94)

    def dense(shift):
        first = 4 * np.arange(ranges) + shift + rng.integers(0, 2, (n, ranges))
        e = np.stack([first, first + rng.integers(0, 2, (n, ranges))], 2).astype(np.uint32).reshape(-1)
        return CRSMatrix(ncols, e, 2 * ranges * np.arange(n + 1, dtype=np.uint64))
    a, b = dense(0), dense(2)
    da, db = ctx.upload(a), ctx.upload(b)
    ctx.reset_stats()
    c = ctx.spadd(da, db)
    launches = ctx.stats()["kernel_launches"]
    same(c.download(), orc.spadd(omat(a), omat(b)), (n, ranges))
    assert (launches == 1) == single, launches
