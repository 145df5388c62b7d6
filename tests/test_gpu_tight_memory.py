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
