"""The work that callers of this package have it do, as cases that can be timed.

Every case goes through the package's public entry points on inputs made by
its own generators.  A matrix result is returned as its row map and entries,
either the device arrays themselves (seen as int64 / int32 tensors, no copy) or
the host arrays, and its nnz.  All results are whole numbers or bytes, exact by
definition, so there is no 64-bit value to hold them against.

Graphs: "small" is the variant-dense generator (a bubble every ~100 bases,
rows of several ranges in the powers), "chromosome" the sparse one (a bubble
every ~830 bases, a few long structural ones).  A graph is an assembly of
contigs -- components of uneven length, as a pangenome has them -- and the seed
gives the order in which they stand, so that the results of two seeds differ in
every row past the first but have the same shape.
"""
import math

import numpy as np
import torch

from diverg_b200 import CRSMatrix, create_distance_index, gen, initialize_runtime

# loci per backbone base of the two generators (SNP and insertion branches add loci)
_LOCI = {"small": 1.0152, "chromosome": 1.0017}


def listed():
    return [
        # one gene- or plasmid-sized component: all launches and host round trips
        {"name": "index_2e3", "kind": "index", "graph": "small", "bases": 2_000, "dmin": 100, "dmax": 300},
        # a 1e5-base region, the plain build of the smaller configuration
        {"name": "index_1e5", "kind": "index", "graph": "small", "bases": 100_000, "dmin": 100, "dmax": 300},
        # windows that start at zero end on a sum instead of a product; odd size
        {"name": "index_zero_1e6", "kind": "index", "graph": "chromosome", "bases": 1_000_003, "dmin": 0, "dmax": 250},
        # the headline: a chromosome-scale build
        {"name": "index_5e7", "kind": "index", "graph": "chromosome", "bases": 50_000_000, "dmin": 400, "dmax": 600},
        # the reference's own call: host matrix in, host index out
        {"name": "index_host_1e6", "kind": "index_host", "graph": "small", "bases": 1_000_000, "dmin": 200,
         "dmax": 500, "u32": False},
        # many components of uneven size with their own windows, built at once
        {"name": "batch_30", "kind": "batch", "graphs": 30, "median": 20_000},
        # one product of a graph's adjacency (the step every power is made of)
        {"name": "spgemm_graph_1e7", "kind": "spgemm_graph", "graph": "chromosome", "bases": 10_000_000},
        # A^k alone, square and multiply over a variant-dense graph
        {"name": "power_1e6", "kind": "power", "graph": "small", "bases": 1_000_000, "k": 100},
        # wide rows: random banded operands, half-width 512, ~4 ranges of ~32 columns a row
        {"name": "spgemm_banded_2e22", "kind": "spgemm_banded", "rows": 1 << 22, "half_width": 512, "mean_ranges": 4.0,
         "mean_len": 32.0},
        {"name": "spadd_banded_2e23", "kind": "spadd_banded", "rows": 1 << 23, "half_width": 512, "mean_ranges": 4.0,
         "mean_len": 32.0},
        # a batch of locus pairs against a resident index
        {"name": "query_1e6", "kind": "query", "graph": "chromosome", "bases": 10_000_000, "dmin": 400, "dmax": 600,
         "pairs": 1_000_000},
        # the adjacency matrix itself, from node lengths and edges
        {"name": "adjacency_1e7", "kind": "adjacency", "graph": "chromosome", "bases": 10_000_000},
    ]


_WINDOWS = ((100, 300), (200, 500), (400, 600), (0, 250), (150, 450), (350, 650))


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi], mostly odd sizes."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("index", "index", "index", "index_host", "batch", "spgemm_graph", "power", "spgemm_banded",
                       "spadd_banded", "query", "adjacency"))
    graph = rng.choice(("small", "chromosome"))
    top = 4_000_000 if graph == "small" else 40_000_000
    dmin, dmax = rng.choice(_WINDOWS)
    if kind == "index":
        return {"kind": kind, "graph": graph, "bases": _log(rng, 1_000, top), "dmin": dmin, "dmax": dmax}
    if kind == "index_host":
        return {"kind": kind, "graph": graph, "bases": _log(rng, 1_000, 2_000_000), "dmin": dmin, "dmax": dmax,
                "u32": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "graphs": rng.randint(2, 31), "median": _log(rng, 1_000, 100_000)}
    if kind == "spgemm_graph" or kind == "adjacency":
        return {"kind": kind, "graph": graph, "bases": _log(rng, 1_000, top)}
    if kind == "power":
        return {"kind": kind, "graph": graph, "bases": _log(rng, 1_000, 4_000_000), "k": rng.randint(2, 300)}
    if kind == "query":
        return {"kind": kind, "graph": graph, "bases": _log(rng, 1_000, top), "dmin": dmin, "dmax": dmax,
                "pairs": _log(rng, 1_000, 4_000_000)}
    return {"kind": kind, "rows": _log(rng, 1_000, 1 << 22), "half_width": rng.choice((128, 256, 512, 700)),
            "mean_ranges": rng.choice((2.0, 4.0, 6.0)), "mean_len": rng.choice((12.0, 20.0, 32.0, 40.0))}


def _make(case):
    return gen.small_graph_spec if case["graph"] == "small" else gen.chromosome_graph_spec


def _contigs(total):
    """6 to 24 contig lengths that add up to `total`, the longest about twice the shortest."""
    m = min(24, max(6, total // 100_000))
    cut = [round(total * k * (2 * m + k - 1) / (m * (3 * m - 1))) for k in range(m + 1)]
    return [cut[k + 1] - cut[k] for k in range(m)]


def _order(n, seed):
    return [int(k) for k in np.random.default_rng(seed).permutation(n)]


def _side_by_side(blocks):
    """The block-diagonal matrix of square blocks."""
    rows = np.cumsum([0] + [b.numRows() for b in blocks])
    ents = np.cumsum([0] + [len(b.entries) for b in blocks])
    rowmap = np.zeros(rows[-1] + 1, np.uint64)
    entries = np.empty(ents[-1], np.uint32)
    for k, b in enumerate(blocks):
        np.add(b.rowmap[1:], np.uint64(ents[k]), out=rowmap[rows[k] + 1:rows[k + 1] + 1])
        np.add(b.entries, np.uint32(rows[k]), out=entries[ents[k]:ents[k + 1]])
    return CRSMatrix(int(rows[-1]), entries, rowmap, sum(b.nnz() for b in blocks))


def _graph(make, bases, seed):
    """The adjacency of an assembly: its contigs in the order that the seed gives."""
    blocks = [gen.graph_adjacency(make(n, seed=100 + k))[0] for k, n in enumerate(_contigs(bases))]
    return _side_by_side([blocks[k] for k in _order(len(blocks), seed)])


def _banded(case, order, salt):
    rows = _contigs(case["rows"])
    return _side_by_side([gen.banded(rows[k], case["half_width"], case["mean_ranges"], case["mean_len"],
                                     seed=salt + 2 * k) for k in order])


def _batch_sizes(case):
    """Log-normal component sizes around the median (sigma 1), spread evenly over the distribution."""
    n = case["graphs"]
    z = [math.sqrt(2.0) * _erfinv(2.0 * (k + 0.5) / n - 1.0) for k in range(n)]
    return [int(min(max(case["median"] * math.exp(v), 1_000), 1_000_000)) for v in z]


def _erfinv(x):
    return float(torch.erfinv(torch.tensor(x, dtype=torch.float64)))


class _Array:
    """A device array of a resident matrix, as torch takes it (keeps the matrix alive)."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr or 0, False), "version": 3,
                                         "strides": None, "stream": None}


def _tensors(m):
    r, e = m.device_arrays()
    return [torch.as_tensor(_Array(m, r, m.nrows + 1, "<i8"), device="cuda"),
            torch.as_tensor(_Array(m, e, m.nentries, "<i4"), device="cuda")
            if m.nentries else torch.empty(0, dtype=torch.int32, device="cuda")]


def prepare(case, seed):
    ctx = initialize_runtime()
    kind = case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind in ("index", "spgemm_graph", "power"):
        s["a"] = ctx.upload(_graph(_make(case), case["bases"], seed))
    elif kind == "index_host":
        a = _graph(_make(case), case["bases"], seed)
        if case["u32"]:
            a = CRSMatrix(a.numCols(), a.entries, a.rowmap.astype(np.uint32), a.nnz(), size_type=np.uint32)
        s["a"] = a
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["graphs"] = [ctx.upload(_graph(gen.small_graph_spec, n, seed + k)) for k, n in enumerate(sizes)]
        s["windows"] = [_WINDOWS[k % 3] for k in range(len(sizes))]
    elif kind in ("spgemm_banded", "spadd_banded"):
        order = _order(len(_contigs(case["rows"])), seed)
        s["a"] = ctx.upload(_banded(case, order, 100))
        s["b"] = ctx.upload(_banded(case, order, 101))
    elif kind == "query":
        a = _graph(_make(case), case["bases"], seed)
        d = ctx.upload(a)
        s["index"] = ctx.distance_index(d, case["dmin"], case["dmax"])
        pairs = gen.query_pairs(a, case["pairs"], 0.5, case["dmin"], case["dmax"], seed=seed)
        s["pairs"] = torch.from_numpy(pairs.view(np.int32)).cuda()
    else:
        parts = [gen.graph_nodes(_make(case)(n, seed=100 + k)) for k, n in enumerate(_contigs(case["bases"]))]
        parts = [parts[k] for k in _order(len(parts), seed)]
        first = np.cumsum([0] + [len(p[0]) for p in parts])
        s["nodes"] = np.concatenate([p[0] for p in parts])
        s["edges"] = np.concatenate([p[1] + np.uint32(first[k]) for k, p in enumerate(parts)])
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "index_host":
        t = create_distance_index(s["a"], case["dmin"], case["dmax"])
        return [t.rowmap.view(np.int32 if case["u32"] else np.int64), t.entries.view(np.int32), t.nnz()]
    if kind == "query":
        out = torch.empty(case["pairs"], dtype=torch.uint8, device="cuda")
        ctx.query_device(s["index"], s["pairs"].data_ptr(), case["pairs"], out.data_ptr())
        return out
    if kind == "batch":
        return [x for m in ctx.batch_distance_index(s["graphs"], s["windows"]) for x in _tensors(m)]
    if kind == "index":
        m = ctx.distance_index(s["a"], case["dmin"], case["dmax"])
    elif kind == "spgemm_graph":
        m = ctx.spgemm(s["a"], s["a"])
    elif kind == "power":
        m = ctx.power(s["a"], case["k"])
    elif kind == "spgemm_banded":
        m = ctx.spgemm(s["a"], s["b"])
    elif kind == "spadd_banded":
        m = ctx.spadd(s["a"], s["b"])
    else:
        m = ctx.adjacency_from_graph(s["nodes"], s["edges"])
    return _tensors(m) + [m.nnz]


def work(case):
    """Bytes of the inputs and outputs, each once: 8 a row for a row map, 8 a
    range; a graph's adjacency and its products hold about a range a row."""
    kind = case["kind"]
    if kind in ("spgemm_banded", "spadd_banded"):
        ranges = case["mean_ranges"] * 0.885  # the generator drops ranges that leave the band or overlap
        out = 1.5 if kind == "spgemm_banded" else 1.55 * ranges
        return {"bytes": case["rows"] * (2 * (8 + 8 * ranges) + 8 + 8 * out), "flops": 0}
    if kind == "batch":
        return {"bytes": 32.0 * _LOCI["small"] * sum(_batch_sizes(case)), "flops": 0}
    n = _LOCI[case["graph"]] * case["bases"]
    if kind == "query":
        return {"bytes": 33.0 * case["pairs"], "flops": 0}
    if kind == "adjacency":
        nodes = case["bases"] * (0.026 if case["graph"] == "small" else 0.0034)
        return {"bytes": 16 * n + 15 * nodes, "flops": 0}
    return {"bytes": 32.0 * n, "flops": 0}
