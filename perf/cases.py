"""Performance cases: the calls that a user of the library makes, each through its public entry point.

A user reorders one matrix (Context.nm_search, or vnm_reorder for the V-block row sort), many matrices
(nm_reorder_batch) or a large one by learned proposals (nm_learned); compresses the result into the V:N:M operand
(SpmmMatrix); multiplies with it, as a plain product (run_async) or inside a graph network (gcn.vnm_spmm, forward and
backward); and trains the proposal network (Mlp.train).  The matrices are the benchmark's kinds: uniform, R-MAT,
Chung-Lu and full V:2:M operands, made from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "vnm-graph-reordering_gb300"))

import vnm_gb300  # noqa: E402
from vnm_gb300 import gcn, learned  # noqa: E402


def listed():
    return [
        # the smallest call: the `spmm` command's search of a 512-row matrix at the command's default 2:8, arrays
        # on the host as the file reader leaves them; latency and launches
        {"name": "search_512", "kind": "search", "graph": "uniform", "rows": 512, "degree": 10, "N": 2, "M": 8,
         "memory": "host"},
        # the headline reorder: find_best over the four schedules, R-MAT, 2:4, the matrix resident in HBM
        {"name": "search_16384", "kind": "search", "graph": "rmat", "rows": 16384, "degree": 16, "N": 2, "M": 4,
         "memory": "device"},
        # the largest exact reorder: the plain search that the learned mode is compared with
        {"name": "search_65536", "kind": "search", "graph": "rmat", "rows": 65536, "degree": 32, "N": 2, "M": 8,
         "memory": "device"},
        # a data set of many small graphs in one call, ragged sizes, packed on the host
        {"name": "batch_256", "kind": "batch", "matrices": 256, "low": 256, "high": 8192, "N": 2, "M": 8, "sched": 0},
        # the V-block row sort between two N:M passes of the `spmm` command
        {"name": "rowsort_16384", "kind": "rowsort", "rows": 16384, "degree": 16, "M": 8, "V": 64},
        # the rest of the command after the search: a fresh operand, multiplied once
        {"name": "operand_16384", "kind": "operand", "graph": "rmat", "order": "degree", "rows": 16384, "degree": 16,
         "M": 4, "V": 64, "n": 128, "dtype": "bf16"},
        # one neighbourhood aggregation of a full-graph network at 256 features, the operand kept
        {"name": "spmm_262144", "kind": "spmm", "graph": "chung_lu", "order": "degree", "rows": 262144, "degree": 20,
         "M": 8, "V": 128, "n": 256, "dtype": "bf16"},
        # a training step's aggregation, forward and backward through two operands, a feature count that needs
        # padding, FP16
        {"name": "gcn_65536", "kind": "gcn", "order": "random", "rows": 65536, "degree": 20, "features": 100,
         "symmetric": False, "dtype": "fp16"},
        # pruned weights (the V:N:M format's intended operand): a 4096-wide layer on a small batch, FP16
        {"name": "structured_4096", "kind": "structured", "rows": 4096, "M": 8, "V": 64, "n": 128, "dtype": "fp16"},
        # and the largest, one row tile for every SM
        {"name": "structured_19456", "kind": "structured", "rows": 19456, "M": 8, "V": 128, "n": 256,
         "dtype": "bf16"},
        # the fast reorder of a large graph: network proposals, run until they stop improving
        {"name": "learned_65536", "kind": "learned", "rows": 65536, "degree": 32, "mode": "network", "targets": 4},
        # fitting the proposal network: 64 Adam steps at the training recipe's batch
        {"name": "train_65536", "kind": "train", "pairs": 65536, "batch": 1024},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: kind, sizes and options over the ranges that the listed cases stand for."""
    kind = rng.choice(["search", "search", "batch", "rowsort", "operand", "operand", "spmm", "spmm", "gcn",
                       "structured", "learned", "train"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    order = rng.choice(["degree", "random"])
    if kind == "search":
        N, M = rng.choice([(2, 4), (2, 8), (2, 8), (1, 4), (4, 8)])
        rows = int(_log(rng, 512, 49152 if (N, M) == (2, 8) else 16384)) // M * M
        return {"kind": kind, "graph": rng.choice(["rmat", "rmat", "uniform"]) if rows <= 4096 else "rmat",
                "rows": rows, "degree": rng.randint(6, 32 if M == 8 else 16), "N": N, "M": M,
                "memory": rng.choice(["host", "device"])}
    if kind == "batch":
        low = int(_log(rng, 128, 1024))
        return {"kind": kind, "matrices": int(_log(rng, 16, 256)), "low": low, "high": int(low * rng.uniform(2, 8)),
                "N": 2, "M": rng.choice([4, 8]), "sched": rng.randrange(4)}
    if kind == "rowsort":
        return {"kind": kind, "rows": int(_log(rng, 1024, 32768)), "degree": rng.randint(4, 20), "M": 8,
                "V": rng.choice([16, 32, 64, 128])}
    if kind == "operand":
        return {"kind": kind, "graph": rng.choice(["rmat", "chung_lu"]), "order": order,
                "rows": int(_log(rng, 2048, 262144)), "degree": rng.randint(4, 32), "M": rng.choice([4, 8]),
                "V": rng.choice([32, 64, 128]), "n": 64 * rng.randint(1, 4), "dtype": dtype}
    if kind == "spmm":
        return {"kind": kind, "graph": rng.choice(["rmat", "chung_lu", "chung_lu"]), "order": order,
                "rows": int(_log(rng, 4096, 262144)), "degree": rng.randint(4, 24), "M": 8, "V": 128,
                "n": 64 * rng.randint(1, 4), "dtype": dtype}
    if kind == "gcn":
        return {"kind": kind, "order": order, "rows": int(_log(rng, 4096, 131072)), "degree": rng.randint(6, 24),
                "features": int(_log(rng, 16, 256)), "symmetric": rng.random() < 0.5, "dtype": dtype}
    if kind == "structured":
        return {"kind": kind, "rows": 128 * int(_log(rng, 8, 152)), "M": rng.choice([4, 8, 8]),
                "V": rng.choice([32, 64, 128]), "n": 64 * rng.randint(1, 4), "dtype": dtype}
    if kind == "learned":
        return {"kind": kind, "rows": int(_log(rng, 4096, 65536)) // 8 * 8, "degree": rng.randint(8, 32),
                "mode": rng.choice(["network", "network", "random", "exhaustive"]), "targets": rng.choice([4, 8, 16])}
    return {"kind": "train", "pairs": int(_log(rng, 4096, 65536)), "batch": rng.choice([256, 512, 1000, 1024])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_held = {}


def _context():
    """The one library handle that a program keeps."""
    if "ctx" not in _held:
        _held["ctx"] = vnm_gb300.Context(0)
    return _held["ctx"]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _split(key, rows):
    return (key // rows).to(torch.int32), (key % rows).to(torch.int32)


def _rmat(rows, edges, g):
    """Symmetrised R-MAT positions (.57, .19, .19, .05), sorted by (row, col), duplicates merged."""
    r = torch.zeros(edges, dtype=torch.int64, device="cuda")
    c = torch.zeros_like(r)
    for _ in range(max(1, math.ceil(math.log2(rows)))):
        u = torch.rand(edges, generator=g, device="cuda", dtype=torch.float64)
        r = 2 * r + (u >= 0.76)
        c = 2 * c + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    r, c = r % rows, c % rows
    return _split(torch.unique(torch.cat([r * rows + c, c * rows + r])), rows)


def _uniform(rows, entries, g):
    return _split(torch.unique(torch.randint(rows * rows, (entries,), generator=g, device="cuda")), rows)


def _chung_lu(rows, degree, g):
    """Symmetrised Chung-Lu positions, power-law exponent 2.1: the first nodes are the hubs."""
    w = torch.arange(1, rows + 1, device="cuda", dtype=torch.float64) ** (-1.0 / 1.1)
    cum = torch.cumsum(w, 0)
    ends = [torch.searchsorted(cum, cum[-1] * torch.rand(rows * degree // 2, generator=g, device="cuda",
                                                         dtype=torch.float64)).clamp_(max=rows - 1) for _ in range(2)]
    return _split(torch.unique(torch.cat([ends[0] * rows + ends[1], ends[1] * rows + ends[0]])), rows)


def _relabelled(row, col, rows, g):
    new = torch.randperm(rows, generator=g, device="cuda")
    key = torch.sort(new[row.long()] * rows + new[col.long()]).values
    return _split(key, rows)


def _values(kind, nnz, g):
    if kind == "normal":
        return torch.randn(nnz, generator=g, device="cuda")
    v = 2.0 * torch.rand(nnz, generator=g, device="cuda") - 1.0  # kept away from 0.00 in two decimals
    return torch.where(v.abs() < 0.005, torch.full_like(v, 0.5), v)


def _graph(case, g):
    rows = case["rows"]
    if case["graph"] == "uniform":
        row, col = _uniform(rows, rows * case["degree"], g)
        val = _values("uniform", len(row), g)
    elif case["graph"] == "rmat":
        row, col = _rmat(rows, rows * case["degree"] // 2, g)
        if case.get("order") == "random":
            row, col = _relabelled(row, col, rows, g)
        val = _values("normal", len(row), g)
    else:  # the symmetric-normalised weights D^-1/2 A D^-1/2
        row, col = _chung_lu(rows, case["degree"], g)
        if case.get("order") == "random":
            row, col = _relabelled(row, col, rows, g)
        d = torch.bincount(row.long(), minlength=rows).clamp_(min=1).double() ** -0.5
        val = (d[row.long()] * d[col.long()]).float()
    return row.contiguous(), col.contiguous(), val.contiguous()


def _batch_rows(case):
    """The batch's row counts: even in their logarithm from low to high, multiples of M, in a mixed order."""
    n, M = case["matrices"], case["M"]
    at = np.random.default_rng(n).permutation(n)
    rows = case["low"] * (case["high"] / case["low"]) ** ((at + 0.5) / n)
    return [-(-int(r) // M) * M for r in rows]


def _entries(key, rows, count, g):
    """Exactly `count` of the sorted positions (uniform ones added where there are too few)."""
    while len(key) < count:
        key = torch.unique(torch.cat([key, torch.randint(rows * rows, (count,), generator=g, device="cuda")]))
    keep = torch.randperm(len(key), generator=g, device="cuda")[:count].sort().values
    return _split(key[keep], rows)


_PAIRS = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


def _structured(case, g):
    """Full V:2:M form: every V x M block keeps 4 columns, every row of it 2 nonzeros among them."""
    rows, M, V = case["rows"], case["M"], case["V"]
    nseg = rows // M
    keep = torch.rand((rows // V, nseg, M), generator=g, device="cuda").argsort(-1)[..., :4].sort(-1).values
    keep = (keep + torch.arange(nseg, device="cuda")[:, None] * M).to(torch.int32)
    pick = torch.tensor(_PAIRS, device="cuda")[torch.randint(6, (rows, nseg), generator=g, device="cuda")]
    cols = torch.empty((rows, nseg, 2), dtype=torch.int32, device="cuda")
    for b in range(rows // V):
        s = slice(b * V, (b + 1) * V)
        cols[s] = torch.gather(keep[b].expand(V, nseg, 4), 2, pick[s])
    row = torch.arange(rows, dtype=torch.int32, device="cuda").repeat_interleave(2 * nseg)
    return row, cols.reshape(-1), torch.randn(2 * rows * nseg, generator=g, device="cuda")


def _half(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float16


def _host(*tensors):
    return tuple(t.cpu().numpy() for t in tensors)


def _spmm_inputs(case, seed):
    g = _gen(seed)
    row, col, val = _structured(case, g) if case["kind"] == "structured" else _graph(case, g)
    B = torch.randn((case["rows"], case["n"]), generator=g, device="cuda").to(_half(case))
    return row, col, val, B


def _gcn_inputs(case, seed):
    g = _gen(seed)
    row, col, val = _graph({"graph": "chung_lu", **case}, g)
    if not case["symmetric"]:  # learned edge weights: one for each direction
        val = _values("uniform", len(row), g)
    X = torch.randn((case["rows"], case["features"]), generator=g, device="cuda")
    G = torch.randn((case["rows"], case["features"]), generator=g, device="cuda")
    return row, col, val, X, G


def _train_inputs(case, seed):
    """Features and gains as the exact scorer's pairs have them, and the network's starting weights."""
    rng = np.random.default_rng(seed)
    n = case["pairs"]
    X = rng.random((n, 32), dtype=np.float32) * rng.random((1, 32), dtype=np.float32)
    X[:, 31] = 1.0
    t = (X @ rng.standard_normal(32).astype(np.float32) + 0.5 * rng.standard_normal(n)).astype(np.float32)
    w = [rng.uniform(-1, 1, s) * a for s, a in ((128 * 32, (6 / 32) ** 0.5), (128, 0), (128 * 128, (6 / 128) ** 0.5),
                                                (128, 0), (128, (3 / 128) ** 0.5), (1, 0))]
    return X, t, np.concatenate(w).astype(np.float32)


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind == "search":
        coo = _graph(case, _gen(seed))
        s["coo"] = _host(*coo) if case["memory"] == "host" else coo
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        mats = []
        for i, rows in enumerate(_batch_rows(case)):
            r, c, v = _graph({"graph": "rmat", "rows": rows, "degree": int(rng.integers(4, 33))},
                             _gen(int(seed) * 1009 + i))
            mats.append((rows,) + _host(r, c, v))
        s["packed"] = vnm_gb300.Context.pack_batch(mats)
    elif kind == "rowsort":
        g, rows = _gen(seed), case["rows"]
        row, col = _rmat(rows, rows * case["degree"], g)
        s["coo"] = _host(*_entries(row.long() * rows + col, rows, rows * case["degree"], g))
    elif kind in ("operand", "spmm", "structured"):
        row, col, val, s["B"] = _spmm_inputs(case, seed)
        if kind == "operand":
            s["coo"] = row, col, val
        else:
            torch.cuda.synchronize()  # the handle works on its own stream
            s["A"] = vnm_gb300.SpmmMatrix(ctx, case["rows"], row, col, val, case["M"], case["V"], case["dtype"])
    elif kind == "gcn":
        row, col, val, X, s["G"] = _gcn_inputs(case, seed)
        s["X"] = X.requires_grad_(True)
        s["A"] = gcn.VnmAdjacency(ctx, case["rows"], row, col, val, M=8, V=128, dtype=case["dtype"],
                                  symmetric=case["symmetric"])
    elif kind == "learned":
        s["coo"] = _graph({"graph": "rmat", **case}, _gen(seed))
        s["net"] = learned.load(ctx, 2, 8) if case["mode"] == "network" else None
        s["seed"] = int(seed) & 0xffff
    else:
        s["X"], s["t"], s["w"] = _train_inputs(case, seed)
        s["net"] = vnm_gb300.Mlp(ctx, 0)
    return s


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "search":
        best, res, newpos = ctx.nm_search(case["rows"], *s["coo"], case["N"], case["M"])
        return {"best": best, "res": res, "newpos": newpos}
    if kind == "batch":
        res, newpos = ctx.nm_reorder_batch(s["packed"], case["N"], case["M"], case["sched"])
        return {"res": res, "newpos": np.concatenate(newpos)}
    if kind == "rowsort":
        out, r, c, newpos = ctx.vnm_reorder(case["rows"], case["rows"], *s["coo"], case["M"], case["V"])
        return {"out": out, "row": r, "col": c, "newpos": newpos}
    if kind == "operand":
        A = vnm_gb300.SpmmMatrix(ctx, case["rows"], *s["coo"], case["M"], case["V"], case["dtype"])
        C = A.run(s["B"])
        A.close()
        return {"C": C}
    if kind in ("spmm", "structured"):
        return {"C": s["A"].run_async(s["B"])}
    if kind == "gcn":
        Y = gcn.vnm_spmm(s["A"], s["X"])
        dX, = torch.autograd.grad(Y, s["X"], s["G"])
        return {"Y": Y.detach(), "dX": dX}
    if kind == "learned":
        mode = {"network": vnm_gb300.LEARNED_MLP, "random": vnm_gb300.LEARNED_RANDOM,
                "exhaustive": vnm_gb300.LEARNED_EXHAUSTIVE}[case["mode"]]
        res, newpos, _ = vnm_gb300.nm_learned(ctx, case["rows"], *s["coo"], 2, 8, mode=mode, net=s["net"],
                                              targets=case["targets"], topk=8, seed=s["seed"])
        return {**res, "newpos": newpos}
    s["net"].set(s["w"])
    loss = s["net"].train(s["X"], s["t"], batch=case["batch"])
    return {"weights": s["net"].get(), "loss": loss}


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "train":
        n, params = case["pairs"] // case["batch"] * case["batch"], 128 * 32 + 128 * 128 + 3 * 128 + 1
        return {"bytes": 4.0 * (33 * n + 2 * params), "flops": 6.0 * n * (128 * 32 + 128 * 128 + 128)}
    if kind == "batch":
        rows = sum(_batch_rows(case))
        return {"bytes": 12.0 * rows * 18 + 4.0 * rows, "flops": 0.0}
    rows = case["rows"]
    nnz = 2.0 * rows * (rows // case["M"]) if kind == "structured" else float(rows * case["degree"])
    if kind in ("search", "learned"):  # the matrix in, a position for every row out
        return {"bytes": 12 * nnz + 4 * rows, "flops": 0.0}
    if kind == "rowsort":  # positions in and out
        return {"bytes": 16 * nnz + 4 * rows, "flops": 0.0}
    if kind == "operand":
        return {"bytes": 12 * nnz + 6.0 * rows * case["n"], "flops": 2 * nnz * case["n"]}
    if kind == "spmm":  # a 32-bit column and value for each entry, B once, C once
        return {"bytes": 8 * nnz + 6.0 * rows * case["n"], "flops": 2 * nnz * case["n"]}
    if kind == "structured":  # 16-bit values and 2-bit places, four columns for each block, B once, C once
        return {"bytes": 2.25 * nnz + 16 * (rows // case["V"]) * (rows // case["M"]) + 6.0 * rows * case["n"],
                "flops": 2 * nnz * case["n"]}
    return {"bytes": 2 * (8 * nnz + 8.0 * rows * case["features"]), "flops": 4 * nnz * case["features"]}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------
def _product64(rows, row, col, val, B):
    crow = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    crow[1:] = torch.cumsum(torch.bincount(row.long(), minlength=rows), 0)
    A = torch.sparse_csr_tensor(crow, col.long(), val.double(), (rows, rows))
    return A @ B.double()


def _train64(X, t, w, batch, lr=1e-3):
    """One epoch of Adam on mean((f(x) - t)^2) / 2; layer inputs and the hidden layers' weights are rounded to
    BF16, as the network is defined."""
    def rounded(x):
        return x.float().bfloat16().double()

    X, t = (torch.from_numpy(a).cuda().double() for a in (X, t))
    p = torch.from_numpy(w).cuda().double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    losses = []
    for k in range(len(X) // batch):
        x, y = rounded(X[k * batch:(k + 1) * batch]), t[k * batch:(k + 1) * batch]
        W1, b1, W2, b2, w3, b3 = torch.split(p, [128 * 32, 128, 128 * 128, 128, 128, 1])
        W1, W2 = rounded(W1.view(128, 32)), rounded(W2.view(128, 128))
        h1 = torch.relu(x @ W1.T + b1)
        h2 = torch.relu(rounded(h1) @ W2.T + b2)
        d = rounded(h2) @ w3 + b3 - y
        losses.append(0.5 * (d * d).mean())
        dy = d / batch
        dz2 = torch.outer(dy, w3) * (h2 > 0)
        dz1 = (dz2 @ W2) * (h1 > 0)
        g = torch.cat([(dz1.T @ x).reshape(-1), dz1.sum(0), (dz2.T @ rounded(h1)).reshape(-1), dz2.sum(0),
                       dy @ rounded(h2), dy.sum().view(1)])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"weights": p, "loss": torch.stack(losses).mean()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("operand", "spmm", "structured"):
        row, col, val, B = _spmm_inputs(case, seed)
        return {"C": _product64(case["rows"], row, col, val, B)}
    if kind == "gcn":
        row, col, val, X, G = _gcn_inputs(case, seed)
        order = torch.argsort(col.long() * case["rows"] + row.long())
        return {"Y": _product64(case["rows"], row, col, val, X),
                "dX": _product64(case["rows"], col[order], row[order], val[order], G)}
    if kind == "train":
        return _train64(*_train_inputs(case, seed), case["batch"])
    return None  # whole numbers
