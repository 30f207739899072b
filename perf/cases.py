"""Performance cases of the counting path.

A case is one call, or one short sequence of calls, that a user of the library
makes on a synthetic graph of a stated shape: a count on a resident graph, an
exact count, a pattern set, a packed collection, or a whole load (edge list in
device memory -> resident graph -> light counts).  Graphs are drawn on the GPU
from the seed: RMAT with (a, b, c, d) = (.57, .19, .19, .05), Erdos-Renyi, and
Chung-Lu with a power-law weight sequence.  `n` need not be a power of two.

Every output is a whole number (counts, raw totals, divisors, flags), so there
is no rounding anywhere and `exact` has nothing to add: outputs must be equal.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fringe-sgc_gb300"))
import fsgc  # noqa: E402

# name -> (vertices, undirected edges): the benchmark's and the tests' patterns
TRI = [(0, 1), (1, 2), (0, 2)]
C4 = [(0, 1), (1, 2), (2, 3), (3, 0)]
K4 = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
C5 = [(0, 1), (1, 2), (2, 3), (3, 4), (4, 0)]
PATTERNS = {
    # vertex and edge cores
    "star_2": (3, [(0, 1), (0, 2)]),
    "star_4": (5, [(0, i) for i in range(1, 5)]),
    "triangle_2_fringes": (5, TRI + [(0, 3), (1, 4)]),
    "triangle_3_on_one": (6, TRI + [(0, 3), (0, 4), (0, 5)]),
    "edge_5_5": (12, [(0, 1)] + [(0, i) for i in range(2, 7)] + [(1, i) for i in range(7, 12)]),
    "edge_3_2_shared": (8, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 5), (1, 6), (0, 7), (1, 7)]),
    # wedge cores whose centre has no fringes
    "wedge_1_on_each_end": (5, [(0, 1), (0, 2), (1, 3), (2, 4)]),
    "wedge_3_1_on_ends": (7, [(0, 1), (0, 2), (1, 3), (1, 4), (1, 5), (2, 6)]),
    "4cycle": (4, C4),
    "4cycle_opposite": (6, C4 + [(0, 4), (2, 5)]),
    # wedge cores with fringes on the centre
    "wedge_centre_and_ends": (6, [(0, 1), (0, 2), (0, 3), (1, 4), (2, 5)]),
    # triangle cores
    "4clique": (4, K4),
    "tailed_4clique_2": (6, K4 + [(0, 4), (0, 5)]),
    "4clique_3_distinct": (7, K4 + [(0, 4), (1, 5), (2, 6)]),
    "triangle_mixed": (7, TRI + [(0, 3), (1, 3), (1, 4), (2, 5), (2, 6)]),
    # general cores
    "5cycle": (5, C5),
    "5cycle_chord_fringe": (6, C5 + [(5, 0), (5, 2)]),
    "house": (5, [(0, 1), (0, 3), (0, 4), (1, 2), (1, 4), (2, 3)]),
    "diamond_2": (6, C4 + [(0, 2), (1, 4), (3, 4), (0, 5), (1, 5), (2, 5)]),
    "4path_ends": (6, [(0, 1), (1, 2), (2, 3), (0, 4), (3, 4), (1, 5)]),
}
# the pattern set of one call on one graph, and the patterns a packed collection is counted with
SET = ["star_2", "star_4", "triangle_2_fringes", "triangle_3_on_one", "edge_5_5", "edge_3_2_shared",
       "wedge_1_on_each_end", "wedge_3_1_on_ends", "4cycle", "4cycle_opposite", "4clique", "tailed_4clique_2",
       "4clique_3_distinct", "triangle_mixed"]
PACKED = ["star_4", "triangle_2_fringes", "edge_5_5", "wedge_1_on_each_end", "4cycle_opposite", "4clique_3_distinct",
          "tailed_4clique_2", "triangle_mixed"]
LOAD = ["star_2", "triangle_2_fringes", "edge_5_5"]


def listed():
    return [
        # the smallest call: the 20,000-vertex ER graph with a triangle and two fringes (launches and read-back)
        {"name": "edge_er20k", "kind": "count", "pattern": "triangle_2_fringes", "family": "er", "n": 20000, "deg": 20.0},
        # edge-core formula with many fringes over a large graph's edges
        {"name": "edge55_rmat20", "kind": "count", "pattern": "edge_5_5", "family": "rmat", "n": 1 << 20, "deg": 32.0},
        # the benchmark's heaviest pattern: endpoint pairs of a wedge, one fringe on each end
        {"name": "wedge_ends_rmat20", "kind": "count", "pattern": "wedge_1_on_each_end", "family": "rmat", "n": 1 << 20,
         "deg": 32.0},
        # the benchmark's 4-cycle with opposite fringes, on a ragged middle-sized graph
        {"name": "wedge_cycle_200k", "kind": "count", "pattern": "4cycle_opposite", "family": "rmat", "n": 200003,
         "deg": 32.0},
        # the benchmark's triangle core with a shared fringe and one on each vertex
        {"name": "triangle_600k", "kind": "count", "pattern": "4clique_3_distinct", "family": "rmat", "n": 600011,
         "deg": 32.0},
        # a triangle core with pairwise and single fringes (all rotations) on a power-law graph of the packed sizes
        {"name": "triangle_mixed_cl", "kind": "count", "pattern": "triangle_mixed", "family": "cl", "n": 50021,
         "deg": 24.0, "exponent": 2.3},
        # per-match family: fringes on the wedge's centre and ends, a graph of the serving mix
        {"name": "wedge_centre_rmat", "kind": "count", "pattern": "wedge_centre_and_ends", "family": "rmat", "n": 3001,
         "deg": 16.0},
        # per-match family: a five-vertex core with a fringe
        {"name": "general_rmat9", "kind": "count", "pattern": "5cycle_chord_fringe", "family": "rmat", "n": 512,
         "deg": 16.0},
        # a graph becomes resident: edge list in device memory, cleaned, prepared, three light counts, released
        {"name": "load_rmat20", "kind": "load", "pattern": "", "family": "rmat", "n": 1 << 20, "deg": 32.0},
        # many patterns on one graph, replayed
        {"name": "set_rmat16", "kind": "set", "pattern": "", "family": "rmat", "n": 1 << 16, "deg": 32.0},
        # many graphs of uneven size in one call per pattern
        {"name": "packed_cl", "kind": "packed", "pattern": "", "family": "cl", "n": 20000, "deg": 20.0, "exponent": 2.4,
         "graphs": 48},
        # the exact 128-bit count beside the u64 one
        {"name": "exact_wedge_100k", "kind": "exact", "pattern": "4cycle_opposite", "family": "rmat", "n": 100003,
         "deg": 32.0},
    ]


# what draw() takes its cases from: (kind, patterns, families, smallest and largest n)
RANGES = [
    ("count", ["star_4", "triangle_2_fringes", "triangle_3_on_one", "edge_5_5", "edge_3_2_shared"],
     ["er", "rmat", "cl"], 300, 1 << 20),
    ("count", ["wedge_1_on_each_end", "wedge_3_1_on_ends", "4cycle", "4cycle_opposite"], ["rmat", "cl", "er"],
     1000, 300000),
    ("count", ["4clique_3_distinct"], ["rmat", "cl"], 1000, 600000),
    ("count", ["4clique", "tailed_4clique_2", "triangle_mixed"], ["rmat", "cl"], 1000, 60000),
    ("count", ["wedge_centre_and_ends"], ["rmat", "cl", "er"], 300, 3000),
    ("count", ["5cycle", "5cycle_chord_fringe", "house", "diamond_2", "4path_ends"], ["rmat", "er"], 100, 500),
    ("load", [""], ["rmat", "cl", "er"], 1000, 1 << 20),
    ("set", [""], ["rmat", "cl"], 1000, 1 << 16),
    ("packed", [""], ["cl"], 1500, 20000),
    ("exact", ["edge_5_5", "wedge_1_on_each_end", "4cycle_opposite", "4clique_3_distinct"], ["rmat", "cl"], 1000, 100000),
]


def draw(rng):
    kind, patterns, families, lo, hi = rng.choice(RANGES)
    family = rng.choice(families)
    small = hi <= 3000
    case = {"kind": kind, "pattern": rng.choice(patterns), "family": family,
            "n": int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))),
            "deg": round(rng.uniform(6.0, 16.0 if small else 32.0), 2)}
    if family == "cl":
        case["exponent"] = round(rng.uniform(2.3, 2.8), 3)
    if kind == "packed":
        case["graphs"] = rng.randint(8, 48)
    return case


# ------------------------------------------------------------------ inputs
def _edges(family, n, deg, exponent, gen):
    """Undirected endpoint pairs, int32 [E, 2] on the GPU: duplicates and loops
    as they fall (the loader drops them)."""
    count = max(1, int(round(n * deg / 2)))
    if family == "er":
        return torch.randint(0, n, (count, 2), generator=gen, device="cuda", dtype=torch.int32)
    if family == "cl":
        w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64).pow(-1.0 / (exponent - 1.0))
        cdf = torch.cumsum(w, 0)
        r = torch.rand((count, 2), generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
        return torch.searchsorted(cdf, r).clamp_(max=n - 1).to(torch.int32)
    scale = max(1, (n - 1).bit_length())
    kept, have = [], 0
    while have < count:  # ids past n are drawn again
        u = torch.zeros(count, device="cuda", dtype=torch.int32)
        v = torch.zeros(count, device="cuda", dtype=torch.int32)
        for _ in range(scale):
            r = torch.rand(count, generator=gen, device="cuda")
            u = u * 2 + (r >= 0.76).to(torch.int32)
            v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).to(torch.int32)
        pairs = torch.stack([u, v], 1)
        pairs = pairs[(u < n) & (v < n)]
        kept.append(pairs)
        have += len(pairs)
    return torch.cat(kept)[:count].contiguous()


def _csr(n, pairs):
    """The cleaned symmetric host CSR of an edge list (packed members are host graphs)."""
    p = pairs.to(torch.int64)
    p = p[p[:, 0] != p[:, 1]]
    key = torch.unique(torch.cat([p[:, 0] * n + p[:, 1], p[:, 1] * n + p[:, 0]]))
    off = torch.searchsorted(key, torch.arange(n + 1, device=key.device, dtype=torch.int64) * n)
    return fsgc.Graph(off.cpu().numpy(), (key % n).to(torch.int32).cpu().numpy())


_context = None


def _ctx():
    """One context per process, as a user's program keeps it."""
    global _context
    if _context is None:
        _context = fsgc.Context(0)
    return _context


class State:
    def __init__(self, kind, names):
        self.kind = kind
        self.names = names
        self.orders = [fsgc.preprocess(*PATTERNS[name]) for name in names]
        self.gid = None
        self.pairs = None
        self.n = 0

    def __del__(self):
        if self.gid is not None:
            _ctx().release(self.gid)


def _member_sizes(n, graphs, rng):
    return [max(1000, int(round(math.exp(rng.uniform(math.log(1000), math.log(max(n, 1001))))))) for _ in range(graphs)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind, n = case["kind"], int(case["n"])
    names = {"set": SET, "packed": PACKED, "load": LOAD}.get(kind, [case["pattern"]])
    s = State(kind, names)
    s.n = n
    ctx = _ctx()
    if kind == "packed":
        sizes = _member_sizes(n, int(case["graphs"]), np.random.default_rng(int(seed)))
        graphs = [_csr(k, _edges(case["family"], k, case["deg"], case.get("exponent", 2.5), gen)) for k in sizes]
        s.gid = ctx.upload_packed(graphs)
        ctx.prepare(s.gid)
        return s
    pairs = _edges(case["family"], n, case["deg"], case.get("exponent", 2.5), gen)
    torch.cuda.synchronize()
    if kind == "load":
        s.pairs = pairs
        return s
    s.gid = ctx.upload_edges(n, (pairs.data_ptr(), len(pairs)), on_device=True)
    ctx.prepare(s.gid)
    return s


# ------------------------------------------------------------------ the calls
def _signed(x):
    """A u64 as the int64 of the same bits."""
    return x - (1 << 64) if x >= 1 << 63 else x


def _rows(results):
    return np.array([[_signed(r.count), _signed(r.raw_total), _signed(r.automorphisms), r.flags, r.core_type]
                     for r in results], dtype=np.int64)


def run(s):
    ctx = _ctx()
    if s.kind == "count":
        return {"results": _rows([ctx.count(s.gid, s.orders[0])])}
    if s.kind == "exact":
        r = ctx.count_exact(s.gid, s.orders[0])
        return {"results": np.array([_signed(r.count_lo), _signed(r.count_hi), _signed(r.raw_lo), _signed(r.raw_hi),
                                     _signed(r.automorphisms), r.flags, r.core_type], dtype=np.int64)}
    if s.kind == "set":
        return {"results": _rows(ctx.count_set(s.gid, s.orders))}
    if s.kind == "packed":
        return {"results": np.stack([_rows(ctx.count_packed(s.gid, mo)) for mo in s.orders])}
    gid = ctx.upload_edges(s.n, (s.pairs.data_ptr(), len(s.pairs)), on_device=True)
    ctx.prepare(gid)
    info = ctx.info(gid)
    results = _rows([ctx.count(gid, mo) for mo in s.orders])
    ctx.release(gid)
    return {"graph": np.array([info.n, info.m, info.max_degree, info.triangles], dtype=np.int64), "results": results}


def work(case):
    """Bytes a pass cannot do without: the graph's offsets (8 bytes) and lists
    (4 bytes an entry) read once per pattern pass that looks at them; a load
    reads the edge list and writes the lists."""
    n, edges = int(case["n"]), float(case["n"]) * case["deg"] / 2
    csr = 8.0 * (n + 1) + 4.0 * 2 * edges
    if case["kind"] == "load":
        return {"bytes": 8.0 * edges + csr, "flops": 0.0}
    if case["kind"] == "packed":
        mean = (n - 1000.0) / math.log(max(n, 1001) / 1000.0)  # of a log-uniform size
        return {"bytes": int(case["graphs"]) * mean / n * csr + 24.0 * int(case["graphs"]), "flops": 0.0}
    return {"bytes": csr, "flops": 0.0}


def exact(case, seed):
    """Counts are whole numbers, compared bit for bit; nothing here is rounded."""
    return None
