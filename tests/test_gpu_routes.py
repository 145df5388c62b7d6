"""GPU: which way a call takes, and what it holds on to: matrices whose caller gave
another column count than the true one, results' memory, chains that do not fit."""
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
