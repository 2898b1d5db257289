"""What the engine's speed is measured on.

A case is one call that a user of the library makes on a grammar-compressed
matrix: a right product Y = M X, a left product y = x^T M, or the way from a
new matrix to its first product (compress, schedule, load, multiply).  The
matrices are the library's two workloads: genotype mosaics (rows = sites,
columns = haplotypes that copy a few founders) and copy-model graphs (row =
node, an adjacency list partly copied from an earlier node's).  They are drawn
here from the seed, so another seed is another matrix and other right-hand
sides, and exact() knows their entries without asking the library.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "g-mm-repair_gb300"))
import gmr  # noqa: E402
from gmr import learn  # noqa: E402

INF = gmr.TROPICAL_INF
INT_MAX = 2**31 - 1
DEV = "cuda:0"


def _mosaic(name, rows, cols, founders, switch, mutation, B, op="right", semiring="plustimes", values=1,
            table="default"):
    c = {"matrix": "mosaic", "op": op, "rows": rows, "cols": cols, "founders": founders, "switch": switch,
         "mutation": mutation, "values": values, "semiring": semiring, "B": B, "table": table}
    return dict(c, name=name) if name else c


def _graph(name, nodes, degree, copy, weighted, B, semiring, table="default"):
    c = {"matrix": "graph", "op": "right", "rows": nodes, "cols": nodes, "degree": degree, "copy": copy,
         "weighted": weighted, "semiring": semiring, "B": B, "table": table}
    return dict(c, name=name) if name else c


def listed():
    return [
        # One vector against a small matrix: an interactive query, where the
        # number of launches is the time.
        _mosaic("vector_small", 2000, 1000, 64, 0.01, 1e-3, 1),
        # One vector, 20,000 sites x 5,000 haplotypes: the smallest of the
        # engine's genotype workloads.
        _mosaic("vector_20k", 20000, 5000, 64, 0.01, 1e-3, 1),
        # One vector, 200,000 x 10,000, a grammar larger than the caches:
        # iterative solvers and score statistics at scale.
        _mosaic("vector_200k", 200000, 10000, 256, 0.005, 5e-4, 1),
        # The batched headline workload: 32 vectors, 200,000 x 10,000, with
        # the learned per-launch table, as the benchmark runs it.
        _mosaic("batch32_200k", 200000, 10000, 256, 0.005, 5e-4, 32, table="learned"),
        # A few vectors at once: block solvers, one value per memory sector.
        _mosaic("batch8_50k", 50000, 5000, 128, 0.005, 1e-3, 8),
        # An odd batch on odd sizes, three dosage values: no lane width
        # divides the rows of X and Y.
        _mosaic("batch33_ragged", 30001, 3001, 96, 0.01, 1e-3, 33, values=3),
        # A wide batch: many phenotypes or a random projection.
        _mosaic("batch128_40k", 40000, 5000, 128, 0.005, 5e-4, 128, table="learned"),
        # One step of 32 breadth-first frontiers, one bit each.
        _graph("frontiers32_8m", 8000000, 24, 0.7, False, 32, "boolean"),
        # One relaxation step of single-source shortest paths.
        _graph("relax_2m", 2000003, 24, 0.7, True, 1, "tropical"),
        # The transposed product for one vector (power iteration uses both).
        _mosaic("left_vector_50k", 50000, 5000, 128, 0.005, 1e-3, 1, op="left"),
        # The transposed product for a batch (Gram products, M^T (M X)).
        _mosaic("left_batch32_50k", 50000, 5000, 128, 0.005, 1e-3, 32, op="left"),
        # From a new matrix to its first product: compression, schedule and
        # load on the GPU, then one vector from host memory.
        _mosaic("compress_20k", 20000, 5000, 64, 0.01, 1e-3, 1, op="compress"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["right"] * 5 + ["left"] * 2 + ["graph"] * 2 + ["compress"])
    table = rng.choice(["default", "default", "learned"])
    if kind == "graph":
        weighted = rng.random() < 0.5
        nodes, degree = _log_int(rng, 50000, 1500000), rng.randint(8, 32)
        copy = round(rng.uniform(0.5, 0.8), 2)
        semiring = rng.choice(["tropical", "boolean"]) if weighted else "boolean"
        B = _log_int(rng, 1, 128) if semiring == "boolean" else _log_int(rng, 1, 8)
        return _graph(None, nodes, degree, copy, weighted, B, semiring, table)
    rows = _log_int(rng, 1000, 100000)
    cols = min(_log_int(rng, 500, 10000), 400000000 // rows)
    founders, switch = _log_int(rng, 32, 256), round(rng.uniform(0.004, 0.012), 4)
    mutation = round(rng.uniform(4e-4, 1.5e-3), 5)
    if kind == "compress":
        rows = min(rows, 20000)
        return _mosaic(None, rows, cols, founders, switch, mutation, 1, op="compress")
    B = _log_int(rng, 1, 128)
    semiring = rng.choice(["plustimes"] * 5 + ["tropical", "boolean"])
    values = 1 if semiring == "boolean" else rng.choice([1, 1, 3])
    if kind == "left":
        return _mosaic(None, rows, cols, founders, switch, mutation, min(B, 64), op="left", semiring=semiring,
                       values=values)
    return _mosaic(None, rows, cols, founders, switch, mutation, B, semiring=semiring, values=values, table=table)


# ------------------------------------------------------------------ matrices
def _values(case):
    """The distinct non-zero values, ascending."""
    if case["matrix"] == "graph":
        return [float(w) for w in range(1, 101)] if case["weighted"] else [1.0]
    return [float(v) for v in range(1, case["values"] + 1)]


def _blocks(case, seed):
    """The matrix of the case.  The one that is compressed in run() has the
    same rows for every seed, in an order drawn from it: the grammar then has
    the same size, so that its arrays can be compared."""
    if case["op"] != "compress":
        yield from _mosaic_blocks(case, seed)
        return
    a = torch.cat([b for _, b in _mosaic_blocks(case, 0)])
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + 53)
    a = a[torch.randperm(case["rows"], generator=g, device=DEV)]
    step = max(1, 32_000_000 // case["cols"])
    for r0 in range(0, case["rows"], step):
        yield r0, a[r0:r0 + step]


def _mosaic_blocks(case, seed):
    """The matrix in blocks of rows on the GPU: uint8 [rows][cols], 0 = no
    entry, v = the v-th value.  Sites draw an allele frequency from
    Beta(1/2, 1/2), founders their allele from it, haplotypes copy a founder,
    switch to another one and mutate."""
    rows, cols, F = case["rows"], case["cols"], case["founders"]
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + 17)
    cur = torch.randint(F, (cols,), generator=g, device=DEV, dtype=torch.int32)
    step = max(1, 32_000_000 // cols)
    for r0 in range(0, rows, step):
        n = min(step, rows - r0)
        at = torch.arange(n, device=DEV, dtype=torch.int32)[:, None]
        last = torch.where(torch.rand((n, cols), generator=g, device=DEV) < case["switch"], at, -1).cummax(0).values
        drawn = torch.randint(F, (n, cols), generator=g, device=DEV, dtype=torch.int32)
        who = torch.where(last >= 0, drawn.gather(0, last.clamp(min=0).long()), cur[None, :])
        cur = who[-1].clone()
        freq = torch.sin(torch.rand((n, 1), generator=g, device=DEV) * (math.pi / 2)) ** 2
        allele = (torch.rand((n, F), generator=g, device=DEV) < freq).to(torch.uint8)
        dose = torch.randint(1, case["values"] + 1, (n, F), generator=g, device=DEV, dtype=torch.uint8)
        flip = torch.rand((n, cols), generator=g, device=DEV) < case["mutation"]
        who = who.long()
        a = (allele * dose).gather(1, who)
        yield r0, torch.where(flip, torch.where(a > 0, 0, dose.gather(1, who)), a)


def _mosaic_codes(case, seed):
    cols = case["cols"]
    parts = []
    for _, a in _blocks(case, seed):
        n = a.shape[0]
        code = torch.zeros((n, cols + 1), dtype=torch.int32, device=DEV)
        code[:, :cols] = (a.to(torch.int32) - 1) * cols + torch.arange(1, cols + 1, dtype=torch.int32, device=DEV)
        keep = torch.ones((n, cols + 1), dtype=torch.bool, device=DEV)
        keep[:, :cols] = a > 0
        parts.append(code[keep].cpu())
    return torch.cat(parts).numpy()


def _graph_entries(case, seed):
    """(row, target, value index) of every edge, by row and target.  Entry i of
    a node is entry i of its prototype with probability `copy`, else a uniform
    target; the smallest weight of a repeated target stays."""
    n, d = case["rows"], case["degree"]
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + 29)
    node = torch.arange(n, device=DEV)
    proto = (torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * node).long().clamp(min=0)
    copies = (torch.rand((n, d), generator=g, device=DEV) < case["copy"])
    copies[0] = False
    target = torch.randint(n, (n, d), generator=g, device=DEV)
    weight = torch.randint(100 if case["weighted"] else 1, (n, d), generator=g, device=DEV)
    who = node[:, None].expand(n, d).clone()
    entry = torch.arange(d, device=DEV)[None, :].expand(n, d)
    for _ in range(64):  # a chain of copies is a few steps long; what is left after 64 draws its own
        on = copies[who, entry]
        if not bool(on.any()):
            break
        who = torch.where(on, proto[who], who)
    key = (target[who, entry] * 128 + weight[who, entry]).sort(1).values
    tgt = key >> 7
    keep = torch.ones((n, d), dtype=torch.bool, device=DEV)
    keep[:, 1:] = tgt[:, 1:] != tgt[:, :-1]
    row = node[:, None].expand(n, d)[keep]
    return row, tgt[keep], (key & 127)[keep]


def _graph_codes(case, seed):
    n = case["rows"]
    row, tgt, w = _graph_entries(case, seed)
    codes = torch.zeros(row.numel() + n, dtype=torch.int32, device=DEV)
    codes[torch.arange(row.numel(), device=DEV) + row] = (w * n + tgt + 1).to(torch.int32)
    return codes.cpu().numpy()


def _rhs(case, seed):
    """X on the GPU: [cols][words], or [rows][words] for the left product."""
    n = case["rows"] if case["op"] == "left" else case["cols"]
    B = case["B"]
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + 41)
    if case["semiring"] == "plustimes":
        return torch.rand((n, B), generator=g, device=DEV) * 2 - 1
    if case["semiring"] == "tropical":  # 1 % of the nodes reached
        x = torch.randint(1001, (n, B), generator=g, device=DEV, dtype=torch.int32)
        return torch.where(torch.rand((n, B), generator=g, device=DEV) < 0.01, x, INT_MAX)
    # 1 %-dense frontiers of a graph; a few sites or haplotypes of a mosaic,
    # whose rows are half full.  Bit b % 32 of word b // 32.
    W, share = (B + 31) // 32, 0.01 if case["matrix"] == "graph" else 2.0 / n
    x = torch.zeros((n, W), dtype=torch.int64, device=DEV)
    for b in range(B):
        x[:, b // 32] |= (torch.rand(n, generator=g, device=DEV) < share).long() << (b % 32)
    return x.to(torch.int32)  # wraps to the same 32 bits


def _csrv(case, seed):
    codes = _graph_codes(case, seed) if case["matrix"] == "graph" else _mosaic_codes(case, seed)
    return gmr.Csrv.from_codes(case["rows"], case["cols"], codes, _values(case))


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    m = _csrv(case, seed)
    X = _rhs(case, seed)
    if case["op"] == "compress":
        return {"case": case, "m": m, "X": X.cpu().numpy()}
    plan = gmr.Plan.build(gmr.repair(m, device=0), case["rows"], case["cols"], device=0)
    eng = gmr.Engine(plan, device=0)
    if case["op"] == "left":
        eng.enable_left(plan)
    elif case["table"] == "learned":
        learn.choose_learned(eng, plan, learn.Mlp.load(learn.MODEL_PATH), case["semiring"], case["B"],
                             mode_model=learn.Mlp.load(learn.MODE_MODEL_PATH))
    Y = torch.empty((case["cols"] if case["op"] == "left" else case["rows"], X.shape[1]), dtype=X.dtype, device=DEV)
    return {"case": case, "eng": eng, "X": X, "Y": Y}


def run(s):
    case = s["case"]
    if case["op"] == "compress":
        g = gmr.repair(s["m"], device=0)
        eng = gmr.Engine(gmr.Plan.build(g, case["rows"], case["cols"], device=0), device=0)
        y = eng.multiply(s["X"], case["semiring"])
        return {"rules": g.rules(), "C": g.C(), "y": y}
    stream = torch.cuda.current_stream().cuda_stream
    if case["op"] == "left":
        s["eng"].multiply_left_device(case["semiring"], s["X"].data_ptr(), s["Y"].data_ptr(), case["B"], stream=stream)
    else:
        s["eng"].multiply_device(case["semiring"], s["X"].data_ptr(), s["Y"].data_ptr(), case["B"], stream=stream)
    return s["Y"]


def exact(case, seed):
    """(+, x) in 64 bits from the uncompressed entries; the other semirings give whole numbers."""
    if case["semiring"] != "plustimes":
        return None
    X = _rhs(case, seed).double()
    if case["matrix"] == "graph":
        row, tgt, w = _graph_entries(case, seed)
        Y = torch.zeros((case["rows"], case["B"]), dtype=torch.float64, device=DEV)
        return Y.index_add_(0, row, (w + 1).double()[:, None] * X[tgt])
    left = case["op"] == "left"
    Y = torch.zeros((case["cols"] if left else case["rows"], case["B"]), dtype=torch.float64, device=DEV)
    for r0, a in _blocks(case, seed):
        a = a.double()
        if left:
            Y += a.T @ X[r0:r0 + a.shape[0]]
        else:
            Y[r0:r0 + a.shape[0]] = a @ X
    return {"rules": None, "C": None, "y": Y.cpu()} if case["op"] == "compress" else Y


def work(case):
    """Bytes: the grammar (8 a rule, 4 a symbol of the top sequence), X and Y,
    each once; compressing also reads the uncompressed string.  Operations: one
    per rule and word, one per symbol and word."""
    nnz, rules, symbols = _sizes(case)
    words = (case["B"] + 31) // 32 if case["semiring"] == "boolean" else case["B"]
    moved = 8 * rules + 4 * symbols + 4 * words * (case["rows"] + case["cols"])
    if case["op"] == "compress":
        moved += 4 * (nnz + case["rows"])
    return {"bytes": moved, "flops": (rules + symbols) * words}


def _sizes(case):
    """Entries, rules and top-sequence symbols of the case's matrix: fits of the
    sizes measured over the ranges above (within 5 %)."""
    if case["matrix"] == "graph":
        nnz = case["rows"] * case["degree"]
        return nnz, 0.195 * case["copy"] * nnz, (1.283 - 1.02 * case["copy"]) * nnz + case["rows"]
    nnz, t = case["rows"] * case["cols"] / 2, case["rows"] / 2000
    several = case["values"] > 1
    return nnz, (2.0 if several else 1.0) * 0.0392 * t**-0.184 * nnz, (2.3 if several else 1.0) * 0.161 * t**-0.0843 * nnz + case["rows"]
