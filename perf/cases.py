"""The workloads by which this runtime's speed is followed.

Each case is one call, or one short program of calls, that a user of the
runtime makes through the Python binding of the C ABI (hyd_cuda.py), on
device-resident arrays.  ``listed()`` holds the workloads of ``bench.py`` and
of the reference's benchmark programs at their own sizes, with the small and
ragged calls beside them; ``draw()`` spreads the same calls over the sizes
between.  ``prepare`` makes the inputs (from the seed alone) and the output
buffers that such a program keeps, ``run`` is one pass, ``work`` the bytes and
operations that the pass cannot do without, and ``exact`` the same results from
plain torch in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "hydrangea-compiler_gb300"))
import hyd_cuda as hc  # noqa: E402

GOLDEN = 0.6180339887498949  # fractional part of the golden ratio: an even spread of sizes
ZIPF_MAX = 256               # longest row of the sparse workloads


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call of an embedding host: one short fused dot, all latency
        {"name": "dot_4099", "op": "dot", "n": 4099},
        # the fused dot of the reference's README at the benchmark's size
        {"name": "dot_2e24", "op": "dot", "n": 1 << 24},
        # weighted histogram of a ragged array over a number of bins that is no power of two
        {"name": "hist_1000_bins", "op": "hist", "n": 20_000_003, "bins": 1000},
        # the headline benchmark's larger bin count
        {"name": "hist_65536_bins", "op": "hist", "n": 1 << 27, "bins": 65536},
        # a fused three-input element chain, the benchmark's memory-bound map
        {"name": "map_zipwith", "op": "map", "n": 1 << 27},
        # exclusive float64 scan at the benchmark's size
        {"name": "scan_f64", "op": "scan", "n": 1 << 27, "dtype": "f64", "reverse": False, "inclusive": False},
        # scanr_inclusive over int64 at a ragged size
        {"name": "scan_i64_ragged", "op": "scan", "n": (1 << 22) + 77, "dtype": "i64", "reverse": True,
         "inclusive": True},
        # segmented_reduce over segments of very uneven length, the benchmark's shape
        {"name": "segreduce_f64", "op": "segreduce", "n": 1 << 27, "max_log2": 16, "dtype": "f64"},
        # heat_2d: iterate of the 5-point clamp stencil on the benchmark's grid
        {"name": "heat_8192", "op": "stencil", "kind": 2, "h": 8192, "w": 8192, "iters": 20},
        # the coo_csr_build program: packed keys, sort_indices, gathers, duplicates summed, CSR
        {"name": "coo_csr_build", "op": "coo_csr", "nnz": 1 << 24, "nrows": 1 << 18, "ncols": 1 << 18, "dup": 4},
        # the spmv program: one CSR matrix of uneven rows, int64 columns
        {"name": "spmv", "op": "spmv", "nrows": 1 << 20, "ncols": 1 << 20, "i32": False},
        # many uneven COO matrices to CSR and SpMV in one call, the benchmark's 512 instances
        {"name": "batched_512", "op": "batched", "ninst": 512, "lo": 10.0, "hi": 18.0},
    ]


def _log(rng, lo, hi):
    """A size spread evenly over the logarithm of [lo, hi]; odd ones as often as even ones."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    op = rng.choice(["dot", "hist", "map", "scan", "segreduce", "stencil", "coo_csr", "spmv", "batched"])
    if op == "dot":
        return {"op": op, "n": _log(rng, 1000, 1 << 26)}
    if op == "hist":
        return {"op": op, "n": _log(rng, 4096, 1 << 27),
                "bins": rng.choice([64, 4096, 65536, _log(rng, 2, 1 << 17)])}
    if op == "map":
        return {"op": op, "n": _log(rng, 4096, 1 << 27)}
    if op == "scan":
        return {"op": op, "n": _log(rng, 1000, 1 << 27), "dtype": rng.choice(["f64", "i64"]),
                "reverse": rng.random() < 0.5, "inclusive": rng.random() < 0.5}
    if op == "segreduce":
        return {"op": op, "n": _log(rng, 4096, 1 << 27), "max_log2": rng.randint(1, 16),
                "dtype": rng.choice(["f64", "i64"])}
    if op == "stencil":
        h, w = _log(rng, 64, 8192), _log(rng, 64, 8192)
        return {"op": op, "kind": rng.choice([1, 2, 3]), "h": h, "w": w, "iters": _log(rng, 1, 20)}
    if op == "coo_csr":
        return {"op": op, "nnz": _log(rng, 4096, 1 << 24), "nrows": _log(rng, 64, 1 << 18),
                "ncols": _log(rng, 64, 1 << 18), "dup": rng.randint(1, 7)}
    if op == "spmv":
        return {"op": op, "nrows": _log(rng, 1000, 1 << 21), "ncols": _log(rng, 1000, 1 << 21),
                "i32": rng.random() < 0.5}
    lo = rng.uniform(8.0, 14.0)
    return {"op": op, "ninst": _log(rng, 1, 256), "lo": lo, "hi": rng.uniform(lo, 18.0)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(n, g, lo=-1.0, hi=1.0):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g).mul_(hi - lo).add_(lo)


def _randint(lo, hi, n, g):
    return torch.randint(lo, hi, (n,), dtype=torch.int64, device="cuda", generator=g)


def _offsets(n, max_log2):
    """Segments of floor(2^U(0, max_log2)) values that cover [0, n): the shape is the case's, whatever the seed."""
    rng = np.random.default_rng(43)
    mean = (2.0 ** max_log2 - 1.0) / (max_log2 * math.log(2.0))
    lens = np.empty(0, dtype=np.int64)
    while lens.sum() < n:
        more = np.floor(2.0 ** rng.uniform(0, max_log2, size=int(n / mean * 1.1) + 16)).astype(np.int64)
        lens = np.concatenate([lens, more])
    cum = np.cumsum(lens)
    k = int(np.searchsorted(cum, n))
    return torch.from_numpy(np.concatenate([[0], cum[:k], [n]]).astype(np.int64)).cuda()


def _zipf_mean():
    k = np.arange(1, ZIPF_MAX + 1, dtype=np.float64)
    return float((k ** -0.5).sum() / (k ** -1.5).sum())


def _row_lengths(nrows, cap, g):
    """Zipf(1.5) row lengths on 1 .. 256, at most `cap` (the row's columns are distinct)."""
    w = torch.arange(1, ZIPF_MAX + 1, dtype=torch.float64, device="cuda") ** -1.5
    cdf = torch.cumsum(w, 0)
    u = torch.rand(nrows, dtype=torch.float64, device="cuda", generator=g) * cdf[-1]
    lens = torch.searchsorted(cdf, u, right=True) + 1
    return torch.minimum(lens.clamp_(max=ZIPF_MAX), cap if torch.is_tensor(cap) else lens.new_tensor(cap))


def _entries(lens, ncols, g):
    """(row of each entry, column of each entry): a row's columns are distinct, in a row order of their own.
    `ncols`: a number, or one per row."""
    nrows = lens.numel()
    start = torch.cumsum(lens, 0) - lens
    row = torch.repeat_interleave(torch.arange(nrows, device="cuda"), lens)
    j = torch.arange(row.numel(), device="cuda") - start[row]
    nc = ncols if torch.is_tensor(ncols) else torch.full((nrows,), ncols, dtype=torch.int64, device="cuda")
    first = (torch.rand(nrows, dtype=torch.float64, device="cuda", generator=g) * nc).long()
    # a stride of nc // len keeps the columns first, first + stride, ... (mod nc) distinct
    return row, (first[row] + j * (nc // lens)[row]) % nc[row]


def _batch_sizes(case):
    n = [int(2.0 ** (case["lo"] + (case["hi"] - case["lo"]) * ((i * GOLDEN) % 1.0))) for i in range(case["ninst"])]
    return np.maximum(np.array(n, dtype=np.int64), ZIPF_MAX)


def prepare(case, seed):
    g, op = _gen(seed), case["op"]
    s = {"op": op}
    if op == "dot":
        s["xs"], s["ys"] = _uniform(case["n"], g), _uniform(case["n"], g)
        s["out"] = torch.zeros(1, dtype=torch.float64, device="cuda")
    elif op == "hist":
        s["data"] = _randint(0, 1 << 20, case["n"], g)
        s["hist"] = torch.zeros(case["bins"], dtype=torch.int64, device="cuda")
    elif op == "map":
        s["xs"] = [_uniform(case["n"], g) for _ in range(3)]
        s["out"] = torch.empty(case["n"], dtype=torch.float64, device="cuda")
    elif op == "scan":
        f64 = case["dtype"] == "f64"
        s["x"] = _uniform(case["n"], g) if f64 else _randint(0, 1 << 40, case["n"], g)
        s["out"] = torch.empty_like(s["x"])
        s["init"] = 0.5 if f64 else 7
        s["reverse"], s["inclusive"] = case["reverse"], case["inclusive"]
    elif op == "segreduce":
        f64 = case["dtype"] == "f64"
        s["offsets"] = _offsets(case["n"], case["max_log2"])
        s["vals"] = _uniform(case["n"], g) if f64 else _randint(-(1 << 40), 1 << 40, case["n"], g)
        s["out"] = torch.empty(s["offsets"].numel() - 1, dtype=s["vals"].dtype, device="cuda")
        s["init"] = 0.0 if f64 else 0
    elif op == "stencil":
        # a simulation goes on from where the last pass left it, on a stream of its own
        s["kind"], s["iters"] = case["kind"], case["iters"]
        s["u"] = _uniform(case["h"] * case["w"], g, 0.0, 1.0).view(case["h"], case["w"])
        s["t"] = torch.empty_like(s["u"])
        s["stream"] = torch.cuda.Stream()
    elif op == "coo_csr":
        nnz, dup = case["nnz"], case["dup"]
        # every `dup` entries share a cell; the cells are distinct (an affine
        # walk over the matrix) until it is full, and the entries shuffled
        cells, rng = case["nrows"] * case["ncols"], np.random.default_rng(int(seed))
        step = next(a for a in rng.integers(1, cells + 1, 1000).tolist() + [1] if math.gcd(a, cells) == 1)
        pick = torch.argsort(torch.rand(nnz, device="cuda", generator=g)) // dup
        cell = (pick % cells * step + int(rng.integers(cells))) % cells
        s["rows"], s["cols"] = cell // case["ncols"], cell % case["ncols"]
        s["vals"] = _randint(-(1 << 40), 1 << 40, nnz, g)
        s["nrows"], s["body"] = case["nrows"], "v = x0 * %dLL + x1;" % case["ncols"]
    elif op == "spmv":
        cap = min(ZIPF_MAX, case["ncols"])
        lens = _row_lengths(case["nrows"], cap, g)
        row, col = _entries(lens, case["ncols"], g)
        key = torch.sort(row * case["ncols"] + col).values
        s["row_ptr"] = torch.cat([lens.new_zeros(1), torch.cumsum(lens, 0)])
        s["col_idx"] = (key % case["ncols"]).to(torch.int32 if case["i32"] else torch.int64)
        s["vals"], s["x"] = _uniform(row.numel(), g), _uniform(case["ncols"], g)
        s["y"] = torch.empty(case["nrows"], dtype=torch.float64, device="cuda")
    else:
        sizes = torch.from_numpy(_batch_sizes(case)).cuda()
        inst = torch.repeat_interleave(torch.arange(sizes.numel(), device="cuda"), sizes)
        base = torch.cumsum(sizes, 0) - sizes
        lens = _row_lengths(inst.numel(), ZIPF_MAX, _gen(4))  # the shapes are the case's, whatever the seed
        row, col = _entries(lens, sizes[inst], g)
        nnz = torch.zeros_like(sizes).index_add_(0, inst, lens)
        # each instance's entries arrive shuffled
        key = torch.randint(0, 1 << 40, (row.numel(),), dtype=torch.int64, device="cuda", generator=g)
        order = torch.argsort(key.add_(inst[row] << 40))
        del key
        row, col = row[order], col[order]
        del order
        s["rows"] = (row - base[inst[row]]).to(torch.int32)
        s["cols"] = col.to(torch.int32)
        del row, col
        s["vals"], s["x"] = _uniform(s["rows"].numel(), g), _uniform(inst.numel(), g)
        s["desc"] = torch.stack([sizes, sizes, nnz], 1).cpu().numpy()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    op = s["op"]
    if op == "dot":
        hc.dot_f64(s["xs"], s["ys"], s["out"])
        return s["out"]
    if op == "hist":
        s["hist"].zero_()  # the `fill [bins] 0` of the program
        hc.weighted_histogram(s["data"], s["hist"])
        return s["hist"]
    if op == "map":
        out, _ = hc.map_f64("v = x0 * x1 + x2;", s["xs"], out=s["out"])
        return out
    if op == "scan":
        hc.scan(s["x"], s["out"], init=s["init"], reverse=s["reverse"], inclusive=s["inclusive"])
        return s["out"]
    if op == "segreduce":
        hc.segmented_reduce(s["offsets"], s["vals"], s["out"], init=s["init"])
        return s["out"]
    if op == "stencil":
        got = hc.iterate_stencil2d(s["kind"], s["u"], s["t"], s["iters"], stream=s["stream"])
        if got is s["t"]:
            s["u"], s["t"] = s["t"], s["u"]
        return got
    if op == "coo_csr":
        rows, cols, vals = s["rows"], s["cols"], s["vals"]
        n = rows.numel()
        keys, perm = torch.empty_like(rows), torch.empty_like(rows)
        hc.map_i64(s["body"], [rows, cols], out=keys)
        hc.sort_indices(keys, perm)
        srows, scols, svals = (torch.empty_like(rows) for _ in range(3))
        for src, dst in ((rows, srows), (cols, scols), (vals, svals)):
            hc.gather(perm, src, dst)
        r, c, v, k = hc.coo_sum_duplicates(srows, scols, svals)
        n = int(k.item())  # the program reads the canonical count
        row_ptr, col_idx, csr_vals = hc.csr_from_sorted_coo(s["nrows"], n, r[:n], c[:n], v[:n])
        return {"perm": perm, "row_ptr": row_ptr, "col_idx": col_idx, "vals": csr_vals, "nnz": n}
    if op == "spmv":
        hc.spmv_csr(s["row_ptr"], s["col_idx"], s["vals"], s["x"], s["y"])
        return s["y"]
    row_ptr, cols, vals, y = hc.batched_coo_csr_spmv(s["desc"], s["rows"], s["cols"], s["vals"], s["x"])
    return {"row_ptr": row_ptr, "cols": cols, "vals": vals, "y": y}


# ---------------------------------------------------------------- least work
def work(case):
    op = case["op"]
    n = case.get("n", 0)
    if op == "dot":
        return {"bytes": 16 * n + 8, "flops": 2 * n}
    if op == "hist":
        return {"bytes": 8 * n + 8 * case["bins"], "flops": 2 * n}
    if op == "map":
        return {"bytes": 32 * n, "flops": 2 * n}
    if op == "scan":
        return {"bytes": 16 * n, "flops": n}
    if op == "segreduce":
        mean = (2.0 ** case["max_log2"] - 1.0) / (case["max_log2"] * math.log(2.0))
        return {"bytes": 8 * n + 16 * (n / mean + 1), "flops": n}
    if op == "stencil":
        points = case["h"] * case["w"]
        return {"bytes": 16 * points, "flops": 6 * points * case["iters"]}
    if op == "coo_csr":
        nnz = case["nnz"]
        k = min(-(-nnz // case["dup"]), case["nrows"] * case["ncols"])
        return {"bytes": 24 * nnz + 8 * nnz + 16 * k + 8 * (case["nrows"] + 1), "flops": nnz}
    mean = _zipf_mean()
    if op == "spmv":
        nr = case["nrows"]
        nnz = nr * mean
        return {"bytes": (12 if case["i32"] else 16) * nnz + 8 * (nr + 1) + 8 * nr + 8 * case["ncols"],
                "flops": 2 * nnz}
    nr = int(_batch_sizes(case).sum())
    nnz = nr * mean
    return {"bytes": 16 * nnz + 12 * nnz + 8 * (nr + case["ninst"]) + 16 * nr, "flops": 2 * nnz}


# ---------------------------------------------------------------- plain torch, 64 bits
def _exact_stencil(s):
    u = s["u"]
    for _ in range(s["iters"]):
        a, b = torch.cat([u[:1], u[:-1]]), torch.cat([u[1:], u[-1:]])
        t = a + b
        t += torch.cat([u[:, :1], u[:, :-1]], 1)
        t += torch.cat([u[:, 1:], u[:, -1:]], 1)
        if s["kind"] == hc.STENCIL_JACOBI:
            u = t / 4.0
        elif s["kind"] == hc.STENCIL_HEAT:
            u = u + 0.1 * (t - 4.0 * u)
        else:
            u = (t + u) / 5.0
    return u


def exact(case, seed):
    s = prepare(case, seed)
    op = s["op"]
    if op == "dot":
        return (s["xs"] * s["ys"]).sum().view(1)
    if op == "map":
        return s["xs"][0] * s["xs"][1] + s["xs"][2]
    if op == "scan" and case["dtype"] == "f64":
        x = s["x"].flip(0) if s["reverse"] else s["x"]
        c = torch.cumsum(x, 0)
        if not s["inclusive"]:
            c = torch.cat([c.new_zeros(1), c[:-1]])
        c += s["init"]
        return c.flip(0) if s["reverse"] else c
    if op == "segreduce" and case["dtype"] == "f64":
        return torch.segment_reduce(s["vals"], "sum", offsets=s["offsets"], initial=0.0) + s["init"]
    if op == "stencil":
        return _exact_stencil(s)
    if op == "spmv":
        row = torch.repeat_interleave(torch.arange(case["nrows"], device="cuda"), s["row_ptr"].diff())
        return torch.zeros_like(s["y"]).index_add_(0, row, s["vals"] * s["x"][s["col_idx"].long()])
    if op == "batched":
        desc = torch.from_numpy(s["desc"]).cuda()
        inst = torch.repeat_interleave(torch.arange(desc.shape[0], device="cuda"), desc[:, 2])
        base = torch.cumsum(desc[:, 0], 0) - desc[:, 0]
        row = s["rows"].long().add_(base[inst])
        col = s["cols"].long().add_(base[inst])
        y = torch.zeros(s["x"].numel(), dtype=torch.float64, device="cuda")
        y.index_add_(0, row, s["vals"] * s["x"][col])
        del inst
        order = torch.argsort((row << 32) + col)
        return {"row_ptr": None, "cols": None, "vals": s["vals"][order], "y": y}
    return None  # whole numbers: held to equality
