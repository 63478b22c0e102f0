"""Performance cases: the work this framework is used for, through its public entry points, on one GPU.

Three kinds of work:
  epoch      one full-batch training epoch (forward, loss, backward, Adam) of a two-layer GCN: `dist1d.Model.train()`
             or `dist2d.Model.train()`, as the gcn_distr*.py scripts run it with one process
  spmm       one product of a cached sparse block with a dense matrix, C = beta*C + A.B: `ops.spmm`, what every stage of
             the 1D / 1.5D / 2D / 3D schedules calls on a rank's block
  spmm_gpu   the drop-in operator on COO indices, C += A.B: `sparse_coo_tensor_cpp.spmm_gpu`, nothing kept between calls
Graphs are the seeded synthetic stand-ins of the datasets: Erdos-Renyi ("er", even degrees) and R-MAT ("rmat", power law),
symmetric, with self loops, normalised by D^-1/2 (A + I) D^-1/2.
"""
import math

import torch

import sparse_coo_tensor_cpp
from cagnet_b200 import datasets, dist1d, dist2d, graphs, ops, partition
from cagnet_b200.backend import CudaBackend


def _epoch(name, graph, n, nnz, f, hidden, classes, train, algorithm="1d", order="reference"):
    case = {"kind": "epoch", "graph": graph, "n": n, "nnz": nnz, "f": f, "hidden": hidden, "classes": classes,
            "train": train, "algorithm": algorithm, "order": order}
    return dict(case, name=name) if name else case


def _spmm(name, graph, n, nnz, parts, f, beta, padded):
    """`n`, `nnz`: the whole graph; the block is the first of `parts` block rows of it (n / parts x n)."""
    case = {"kind": "spmm", "graph": graph, "n": n, "nnz": nnz, "parts": parts, "f": f, "beta": beta, "padded": padded}
    return dict(case, name=name) if name else case


def _spmm_gpu(name, graph, n, nnz, parts, f):
    case = {"kind": "spmm_gpu", "graph": graph, "n": n, "nnz": nnz, "parts": parts, "f": f}
    return dict(case, name=name) if name else case


def listed():
    return [
        # citation-network size (Cora): everything fits in L2, launches and host time are the cost
        _epoch("epoch_citation", "er", 2708, 13540, 1433, 16, 7, 0.3),
        # the small even-degree benchmark graph (16,384 vertices, degree 16)
        _epoch("epoch_er16k", "er", 16384, 278528, 128, 16, 8, 1.0),
        # a mid-size power-law graph through the 2D script on one GPU, sizes that divide nothing
        _epoch("epoch_mid_2d", "rmat", 65521, 3200000, 300, 16, 24, 0.66, algorithm="2d"),
        # a product co-purchase graph, wider hidden layer, sparse products at the narrower width
        _epoch("epoch_products_min_width", "rmat", 300007, 20000000, 100, 64, 47, 0.5, order="min_width"),
        # a protein-similarity sample: few features, many classes, so the backward product is the wide one
        _epoch("epoch_protein", "rmat", 700001, 24000000, 128, 16, 256, 1.0),
        # the headline benchmark: Reddit's shape, 493 nonzeros per row, 602 features
        _epoch("epoch_reddit", "rmat", 232965, 114600000, 602, 16, 41, 0.66),
        # one small product on its own: launch latency
        _spmm("spmm_small_w16", "er", 2708, 13540, 1, 16, 0, True),
        # sparse power-law graph at the hidden width
        _spmm("spmm_rmat20_w16", "rmat", 1048576, 32400000, 1, 16, 0, True),
        # odd width in a caller's own contiguous layout (rows not 16-byte aligned), added to what is there
        _spmm("spmm_rmat_w41_add", "rmat", 500009, 16000000, 1, 41, 1, False),
        # sparse power-law graph at the feature width: B is far larger than L2
        _spmm("spmm_rmat20_w602", "rmat", 1048576, 32400000, 1, 602, 0, True),
        # a rank's block row in an 8-GPU run of a dense power-law graph
        _spmm("spmm_rank_block_w256", "rmat", 180001, 60000000, 8, 256, 0, True),
        # the drop-in operator as the reference's own scripts would call it on a block (indices checked each call)
        _spmm_gpu("spmm_gpu_block_w128", "rmat", 262139, 8000000, 2, 128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["epoch"] * 5 + ["spmm"] * 5 + ["spmm_gpu"] * 2)
    graph = rng.choice(["er", "rmat", "rmat"])
    n = _log(rng, 2500, 1050000)
    degree = _log(rng, 4, 500)
    # at most 60 M nonzeros, and never denser than a sixteenth of the matrix (R-MAT does not fill up further)
    nnz = n + max(n, min(n * degree, 60000000 - n, n * n // 16))
    if kind == "epoch":
        f = max(8, min(_log(rng, 16, 1433), 600000000 // n, 35000000000 // nnz))
        classes = _log(rng, 3, 256)
        if nnz > 30000000:
            classes = min(classes, 128)
        algorithm, order = rng.choice([("1d", "reference"), ("1d", "reference"), ("2d", "reference"), ("1d", "min_width")])
        return _epoch(None, graph, n, nnz, f, rng.choice([16, 16, 32, 64]), classes, rng.choice([0.3, 0.66, 1.0]),
                      algorithm, order)
    f = max(4, min(_log(rng, 4, 700), 35000000000 // nnz))
    parts = rng.choice([1, 1, 2, 4, 8])
    if kind == "spmm":
        return _spmm(None, graph, n, nnz, parts, f, rng.choice([0, 0, 1]), rng.random() < 0.75)
    if nnz > 20000000:
        parts = max(parts, 4)
    return _spmm_gpu(None, graph, n, nnz, parts, f)


def _spec(case, f, classes, train):
    n, nnz = case["n"], case["nnz"]
    size = "deg=%d" % max(1, round((nnz - n) / n)) if case["graph"] == "er" else "nnz=%d" % nnz
    return "%s:n=%d,%s,f=%d,c=%d,train=%g" % (case["graph"], n, size, f, classes, train)


def _block(case, seed):
    """The first block row of the normalised adjacency matrix cut into case["parts"], as a rank holds it."""
    n = case["n"]
    _, edges, _, _, _, _ = datasets.load(_spec(case, 1, 2, 1.0), device="cuda", seed=seed)
    adj = graphs.add_self_loops(edges, n)
    _, blocks = partition.oned_partition(0, case["parts"], torch.empty(n, 1, device="cuda"), adj, True)
    return partition.fuse_columns(blocks)


def prepare(case, seed):
    torch.cuda.set_device(0)
    be = CudaBackend()
    if case["kind"] == "epoch":
        x, edges, data, f, classes, _ = datasets.load(_spec(case, case["f"], case["classes"], case["train"]),
                                                      device="cuda", seed=seed)
        adj = graphs.add_self_loops(edges, case["n"])
        if case["algorithm"] == "2d":
            model = dist2d.Model(dist2d.Runtime(be), 0, 1, x, adj, data, f, classes)
        else:
            model = dist1d.Model(dist1d.Runtime(be, order=case["order"]), 0, 1, x, adj, data, f, classes)
        model.init_weights(case["hidden"])
        return {"case": case, "model": model}
    block = _block(case, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    B = torch.randn(block.n_cols, case["f"], generator=g, device="cuda")
    C = torch.randn(block.n_rows, case["f"], generator=g, device="cuda")
    if case["kind"] == "spmm":
        if case["padded"]:
            B, C = ops.to_padded(B), ops.to_padded(C)
        return {"case": case, "block": be.make_block(block), "B": B, "C": C}
    return {"case": case, "rows": block.rows.int(), "cols": block.cols.int(), "vals": block.vals, "n": block.n_rows,
            "m": block.n_cols, "B": B, "C": C}


def run(state):
    case = state["case"]
    if case["kind"] == "epoch":
        model = state["model"]
        out = model.train()
        return {"out": out, "loss": model.last_loss, "grad_w1": model.weight1.grad, "grad_w2": model.weight2.grad}
    if case["kind"] == "spmm":
        return ops.spmm(state["block"], state["B"], state["C"], float(case["beta"]))
    sparse_coo_tensor_cpp.spmm_gpu(state["rows"], state["cols"], state["vals"], state["n"], state["m"], state["B"],
                                   state["C"])
    return state["C"]


def work(case):
    """Matrices and indices once each: adjacency as offsets + (index, value) pairs, dense operands and results in fp32."""
    n, nnz, f = case["n"], case["nnz"], case["f"]
    if case["kind"] == "epoch":
        h, c = case["hidden"], case["classes"]
        # widths of the sparse products: layer 1 forward and backward, layer 2 forward and backward
        if case["order"] == "min_width":
            sparse = (2 * h if h <= f else f) + 2 * min(h, c)
        else:
            sparse = f + h + h + c
        dense = 2 * f * h + 3 * h * c
        weights = f * h + h * c
        # adjacency, features, labels and mask in; log-probabilities and gradients out; Adam reads and writes
        # the weights and both moments
        nbytes = 8 * nnz + 4 * (n + 1) + 4 * n * f + 9 * n + 4 * n * c + 4 * weights * 7
        return {"bytes": nbytes, "flops": 2 * nnz * sparse + 2 * n * dense}
    rows, nnz = -(-n // case["parts"]), nnz / case["parts"]
    accumulates = case["kind"] == "spmm_gpu" or case["beta"] != 0
    nbytes = 4 * n * f + 4 * rows * f * (2 if accumulates else 1)
    nbytes += 12 * nnz if case["kind"] == "spmm_gpu" else 8 * nnz + 4 * (rows + 1)
    return {"bytes": nbytes, "flops": 2 * nnz * f}


def tolerance(case):
    # fp32 sums in another order.  An epoch's weight gradients add up signed terms that cancel to about a thousandth of
    # their size, which magnifies the rounding of the sums below them.
    return {"rel": 1e-4} if case["kind"] == "epoch" else {"rel": 1e-5}
