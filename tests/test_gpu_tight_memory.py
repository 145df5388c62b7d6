"""GPU: calls that fit the device's memory by a little.  Working memory that only makes
a call faster must not be what its result lacks.  Each test runs in a process of its
own, in which torch holds all but a given part of the memory."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

START = """
import sys, time
sys.path.insert(0, %r)
import numpy as np, torch
from diverg_b200 import CRSMatrix, gen
from diverg_b200.runtime import Context
ctx = Context(0)

def leave(free):
    # all but `free` bytes of the device's memory
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")
    time.sleep(1.2)  # (the context asks for the free memory once a second)
    assert abs(torch.cuda.mem_get_info()[0] - free) < 64 << 20
    return hog
""" % ROOT


def child(code):
    r = subprocess.run([sys.executable, "-c", START + code], capture_output=True, text=True, timeout=300,
                       cwd=ROOT, env=dict(os.environ))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_a_product_that_fits_in_range_crs():
    # 2e7 rows: the chain's arena, two slot matrices and the result are 1.35 GB, in range
    # CRS the product takes 0.5
    child("""
n = 20_000_000
i = np.arange(n - 1, dtype=np.uint32) + 1
a = CRSMatrix(n, np.stack([i, i], 1).reshape(-1), 2 * np.minimum(np.arange(n + 1, dtype=np.uint64), n - 1), n - 1)
small, _ = gen.graph_adjacency(gen.small_graph_spec(30_000, seed=91))
s = ctx.upload(small)
ctx.spgemm(s, s).free()  # (kernels are loaded)
d = ctx.upload(a)
hog = leave(1_000_000_000)
c = ctx.spgemm(d, d)
del hog
m = c.download()
assert np.array_equal(m.rowmap, 2 * np.minimum(np.arange(n + 1, dtype=np.uint64), n - 2))
assert np.array_equal(m.entries, np.stack([i[1:], i[1:]], 1).reshape(-1)) and m.nnz() == n - 2
""")


def test_a_long_range_product_without_its_tables():
    # 2^19 rows of one range of 400 columns: the result is 1.57 GB, the tables of unions
    # of B's rows 0.25, which no longer fit beside it
    child("""
n = 1 << 19
i = np.arange(n, dtype=np.int64)
a = CRSMatrix(n, np.stack([i, np.minimum(i + 399, n - 1)], 1).astype(np.uint32).reshape(-1),
              2 * np.arange(n + 1, dtype=np.uint64))
# row j: the columns c of [j, j + 350] with c = 2 (j mod 20) modulo 40; never neighbours
first = i + (2 * (i % 20) - i) % 40
cols = first[:, None] + 40 * np.arange(9)
ok = (cols <= i[:, None] + 350) & (cols < n)
rm = np.concatenate(([0], np.cumsum(2 * ok.sum(1)))).astype(np.uint64)
b = CRSMatrix(n, np.repeat(cols[ok], 2).astype(np.uint32), rm)
da, db = ctx.upload(a), ctx.upload(b)
w = gen.banded(1 << 15, 512, 4.0, 80.0, seed=92)
dw = ctx.upload(w)
ctx.spgemm(dw, dw).free()  # (kernels are loaded: these name enough rows for tables)
dw.free()
ctx.trim()
hog = leave(1_740_000_000)
c = ctx.spgemm(da, db)
del hog
ctx.trim()
m = c.download()
for j in [0, 1, 63, 64, n // 2 + 5, n - 400, n - 1] + list(range(100_000, 100_040)):
    want = np.unique(cols[j:j + 400][ok[j:j + 400]])
    e = m.entries[int(m.rowmap[j]):int(m.rowmap[j + 1])].reshape(-1, 2)
    assert np.array_equal(e[:, 0], want) and np.array_equal(e[:, 1], want), j
assert m.entries.size > 700 * n and m.nnz() == m.entries.size // 2
""")


def test_an_adjacency_matrix_of_many_edges_in_a_row():
    # 1e4 nodes of one base with an edge to every later one: 5e7 edges, 0.60 GB, and one
    # range a row.  A range an edge would be 0.40 GB more
    child("""
n = 10_000
def edges(n):
    u = np.repeat(np.arange(1, n, dtype=np.uint32), np.arange(n - 1, 0, -1))
    at = np.concatenate(([0], np.cumsum(np.arange(n - 1, 0, -1)))).astype(np.int64)
    v = (np.arange(u.size) - at[u - 1]).astype(np.uint32) + u + 1
    return np.stack([u, v], 1)
ctx.adjacency_from_graph(np.ones(100, np.uint32), edges(100)).free()  # (kernels are loaded)
e = edges(n)
hog = leave(800_000_000)
a = ctx.adjacency_from_graph(np.ones(n, np.uint32), e)
del hog
m = a.download()
i = np.arange(n - 1, dtype=np.uint32)
assert np.array_equal(m.rowmap, 2 * np.minimum(np.arange(n + 1, dtype=np.uint64), n - 1))
assert np.array_equal(m.entries.reshape(-1, 2), np.stack([i + 1, np.full(n - 1, n - 1, np.uint32)], 1))
assert m.nnz() == len(e)
""")
