"""Performance cases of the framework: what its users have it compute, at the sizes they use.

``listed()`` holds the named cases, ``draw()`` makes further ones over the same ranges.  A case is a dict of plain
values; ``prepare()`` builds what a caller holds before the call (device tensors, a matrix handle, a compiled
module, numpy arrays for the calls that take numpy arrays), ``run()`` is one pass through the public entry points.

Operations (``op``):
  spmv_call   ``KokkosBackend.compile(...).spmv`` on numpy arrays: the calling convention of a generated module
  spmv        ``CsrMatrix.spmv`` with everything resident on the device
  spmm        ``CsrMatrix.spmm`` (``format`` csr) or ``spmm_dcsr`` (``format`` dcsr), fp64
  bspmm       ``bspmm_csrv``: batched SpMM over a CSRV tensor, fp32
  gemm        ``bgemm``: C += A B in fp32, one product (``batch`` 1) or a batch of them
  pcg         ``CsrMatrix.pcg`` on the 5-point Laplacian, resident, a fixed number of iterations
  pcg_call    ``KokkosBackend.compile(...).pcg`` on numpy arrays, to a tolerance
  mht         ``CsrMatrix.mht``: hitting-time moments of a grid graph, a fixed number of iterations per solve
"""
import functools
import math

import torch

from lapis_b200 import KokkosBackend, device, modules

DEV = "cuda"


def listed():
    return [
        # examples/spmv.py: a module compiled once and called with numpy arrays; 10,000 rows of 10 entries
        {"name": "spmv_call_10k", "op": "spmv_call", "rows": 10_000, "mean": 10, "idx": 64},
        # the same matrix held on the device by a loop that calls SpMV over and over: launches and latency
        {"name": "spmv_10k", "op": "spmv", "rows": 10_000, "dist": "uniform", "mean": 10, "idx": 64, "tune": "none", "accumulate": True},
        # a large graph: skewed rows, columns all over a vector that does not fit L1, 1.3e8 entries
        {"name": "spmv_8m_skewed", "op": "spmv", "rows": 1 << 23, "dist": "power", "mean": 16, "idx": 64, "tune": "relaxed", "accumulate": False},
        # a block of 64 right-hand sides against a large matrix
        {"name": "spmm_2m_k64", "op": "spmm", "format": "csr", "rows": 1 << 21, "dist": "uniform", "mean": 32, "k": 64, "idx": 64, "accumulate": False},
        # doubly compressed storage, ragged rows, an odd number of right-hand sides, 32-bit indices
        {"name": "spmm_dcsr_ragged_k37", "op": "spmm", "format": "dcsr", "rows": 50_021, "dist": "power", "mean": 16, "k": 37, "idx": 32, "accumulate": True},
        # message passing with 8 edge channels and 64 features per node (examples/bspmm.py at working size)
        {"name": "bspmm_131k_8x64", "op": "bspmm", "rows": 1 << 17, "mean": 32, "nh": 8, "dh": 64, "idx": 32},
        # benchmarks/gemm: one large square product
        {"name": "gemm_8192", "op": "gemm", "batch": 1, "m": 8192, "n": 8192, "k": 8192},
        # benchmarks/batched_gemm: thousands of small square products
        {"name": "bgemm_4096x128", "op": "gemm", "batch": 4096, "m": 128, "n": 128, "k": 128},
        # a layer whose sizes are multiples of nothing
        {"name": "gemm_ragged_1000", "op": "gemm", "batch": 1, "m": 1000, "n": 1501, "k": 777},
        # a large elliptic solve, 200 iterations
        {"name": "pcg_4096sq", "op": "pcg", "grid": 4096, "idx": 32, "iters": 200},
        # examples/pcg_solve.py: a small system solved to a tolerance through the compiled module
        {"name": "pcg_call_32sq", "op": "pcg_call", "grid": 32, "idx": 32},
        # examples/hitting_times.py on a large grid graph: two solves with the masked Laplacian
        {"name": "mht_2048sq", "op": "mht", "grid": 2048, "idx": 32, "iters": 40},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["spmv_call", "spmv", "spmv", "spmm", "spmm", "bspmm", "gemm", "gemm", "gemm", "pcg", "pcg_call", "mht"])
    idx = rng.choice([32, 64])
    if op == "spmv_call":
        return {"op": op, "rows": _log(rng, 1000, 300_000), "mean": rng.randint(3, 24), "idx": idx}
    if op == "spmv":
        dist = rng.choice(["uniform", "power", "grid"])
        rows, mean = _log(rng, 10_000, 1 << 23), rng.randint(4, 32)
        if dist == "grid":
            rows, mean = math.isqrt(rows) ** 2, 5
        return {"op": op, "rows": min(rows, (1 << 27) // mean), "dist": dist, "mean": mean, "idx": idx,
                "tune": rng.choice(["none", "strict", "relaxed"]), "accumulate": rng.random() < 0.5}
    if op == "spmm":
        k, mean = _log(rng, 2, 130), rng.randint(4, 40)
        rows = _log(rng, 10_000, min(1 << 21, (1 << 27) // k, (1 << 32) // (k * mean)))
        return {"op": op, "format": rng.choice(["csr", "dcsr"]), "rows": rows, "dist": rng.choice(["uniform", "power"]), "mean": mean,
                "k": k, "idx": idx, "accumulate": True if rng.random() < 0.5 else False}
    if op == "bspmm":
        nh, dh, mean = rng.randint(1, 16), _log(rng, 4, 128), rng.randint(4, 40)
        return {"op": op, "rows": _log(rng, 4000, min(1 << 18, (1 << 26) // (nh * dh), (1 << 31) // (nh * dh * mean))), "mean": mean,
                "nh": nh, "dh": dh, "idx": idx}
    if op == "gemm":
        batch = 1 if rng.random() < 0.5 else _log(rng, 2, 4096)
        lo, hi = (32, 8192) if batch == 1 else (4, 256)
        m, n, k = (_log(rng, lo, hi) for _ in range(3))
        if rng.random() < 0.5:
            m, n, k = -(-m // 128) * 128, -(-n // 128) * 128, -(-k // 32) * 32
        return {"op": op, "batch": max(1, min(batch, (1 << 26) // max(m * n, n * k, m * k))), "m": m, "n": n, "k": k}
    if op == "pcg":
        grid = _log(rng, 64, 4096)
        return {"op": op, "grid": grid, "idx": idx, "iters": rng.randint(20, min(200, 2 * grid))}
    if op == "pcg_call":
        return {"op": op, "grid": _log(rng, 10, 250), "idx": idx}
    return {"op": op, "grid": _log(rng, 64, 2048), "idx": idx, "iters": rng.randint(20, 60)}


# ---- inputs, made on the device ----------------------------------------------------------------------------------
def _idx(case):
    return torch.int32 if case["idx"] == 32 else torch.int64


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(gen, shape, dtype=torch.float64, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, dtype=dtype, device=DEV) * (hi - lo) + lo


def _power_law_lengths(n, mean, cap, gen):
    """Row lengths with density ~ L^-2 on [x, cap], x solved so that the mean is ``mean``."""
    lo, hi = 1e-6, float(cap)
    for _ in range(100):
        x = 0.5 * (lo + hi)
        lo, hi = (x, hi) if math.log(cap / x) / (1.0 / x - 1.0 / cap) < mean else (lo, x)
    u = torch.rand(n, generator=gen, dtype=torch.float64, device=DEV)
    return (1.0 / (1.0 / x - u * (1.0 / x - 1.0 / cap))).round().clamp_(1, cap).to(torch.int64)


def _random_csr(rows, cols, dist, mean, dtype, gen):
    """CSR with distinct ascending columns spread evenly at random over each row (entry j of a row of L entries lies
    in the j-th of L equal parts of the columns)."""
    if dist == "power":
        lens = _power_law_lengths(rows, mean, min(4096, cols), gen)
    else:
        lens = torch.full((rows,), min(mean, cols), dtype=torch.int64, device=DEV)
    pos = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=pos[1:])
    nnz = int(pos[-1])
    j = torch.arange(nnz, device=DEV) - torch.repeat_interleave(pos[:-1], lens)
    lens = torch.repeat_interleave(lens, lens)
    start = j * cols // lens
    width = (j + 1) * cols // lens - start
    del j, lens
    crd = (start + (torch.rand(nnz, generator=gen, dtype=torch.float64, device=DEV) * width).to(torch.int64)).to(dtype)
    return pos.to(dtype), crd


def _laplacian(g, dtype, diagonal=True):
    """5-point stencil on a g x g grid, Dirichlet boundary; without its diagonal: the grid graph's adjacency."""
    n = g * g
    row = torch.arange(n, device=DEV)
    i, j = row // g, row % g
    yes = torch.ones(n, dtype=torch.bool, device=DEV)
    parts = [(i > 0, -g, -1.0), (j > 0, -1, -1.0), (yes, 0, 4.0), (j < g - 1, 1, -1.0), (i < g - 1, g, -1.0)]
    if not diagonal:
        parts = [(m, o, 1.0) for m, o, _ in parts if o != 0]
    there = torch.stack([m for m, _, _ in parts], 1)
    pos = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(there.sum(1), 0, out=pos[1:])
    crd = torch.stack([(row + o).to(dtype) for _, o, _ in parts], 1)[there]
    val = torch.tensor([v for _, _, v in parts], dtype=torch.float64, device=DEV).expand(n, len(parts))[there]
    return pos.to(dtype), crd, val


def _grid_nnz(g, diagonal=True):
    return (5 if diagonal else 4) * g * g - 4 * g


@functools.lru_cache(maxsize=None)
def _module(op, idx):
    """Compiled once per program, as a user does."""
    enc = modules.CSR32 if idx == 32 else modules.CSR64
    text = modules.spmv(enc) if op == "spmv_call" else modules.pcg(enc)
    return KokkosBackend.KokkosBackend(decompose_tensors=True).compile(text)


def prepare(case, seed):
    op, gen = case["op"], _gen(seed)
    s = {"case": case}
    if op in ("spmv_call", "spmv"):
        rows = case["rows"]
        if case.get("dist") == "grid":
            g = math.isqrt(rows)
            rows = g * g
            pos, crd, val = _laplacian(g, _idx(case))
        else:
            pos, crd = _random_csr(rows, rows, case.get("dist", "uniform"), case["mean"], _idx(case), gen)
            val = _uniform(gen, crd.numel())
        x, y = _uniform(gen, rows), _uniform(gen, rows)
        if op == "spmv_call":
            s["args"] = [t.cpu().numpy() for t in (pos, crd, val)] + [((rows, rows), (pos.numel(), crd.numel(), val.numel()))] + [
                t.cpu().numpy() for t in (x, y)]
            s["fn"] = _module(op, case["idx"]).spmv
            return s
        s["A"] = device.CsrMatrix(pos, crd, val, (rows, rows))
        if case["tune"] != "none":
            s["A"].tune(relaxed=case["tune"] == "relaxed")
        s["x"], s["y"] = x, y
    elif op == "spmm":
        rows, k = case["rows"], case["k"]
        pos, crd = _random_csr(rows, rows, case["dist"], case["mean"], _idx(case), gen)
        val = _uniform(gen, crd.numel())
        s["B"] = _uniform(gen, (rows, k))
        if case["format"] == "csr":
            s["A"] = device.CsrMatrix(pos, crd, val, (rows, rows))
            s["C"] = _uniform(gen, (rows, k))
        else:  # every other row of C is stored in A
            s["A"] = (torch.arange(0, 2 * rows, 2, device=DEV, dtype=_idx(case)), pos, crd, val)
            s["C"] = _uniform(gen, (2 * rows, k))
    elif op == "bspmm":
        n, nh, dh = case["rows"], case["nh"], case["dh"]
        pos, crd = _random_csr(n, n, "uniform", case["mean"], _idx(case), gen)
        s["A"] = (pos, crd, _uniform(gen, crd.numel() * nh, torch.float32))
        s["B"] = _uniform(gen, (n, dh, nh), torch.float32)
    elif op == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        lead = (b,) if b > 1 else ()
        s["A"], s["B"], s["C"] = (_uniform(gen, lead + d, torch.float32) for d in ((m, k), (k, n), (m, n)))
    elif op in ("pcg", "pcg_call"):
        g = case["grid"]
        pos, crd, val = _laplacian(g, _idx(case))
        b, dinv = _uniform(gen, g * g, lo=0.0), torch.full((g * g,), 0.25, dtype=torch.float64, device=DEV)
        if op == "pcg":
            s["A"] = device.CsrMatrix(pos, crd, val, (g * g, g * g), tune=True)
            s["b"], s["dinv"] = b, dinv
        else:
            s["args"] = [t.cpu().numpy() for t in (pos, crd, val)] + [((g * g, g * g), (pos.numel(), crd.numel(), val.numel()))] + [
                t.cpu().numpy() for t in (b, dinv)] + [1e-6, 2000]
            s["fn"] = _module(op, case["idx"]).pcg
    elif op == "mht":
        g = case["grid"]
        pos, crd, val = _laplacian(g, _idx(case), diagonal=False)
        s["A"] = device.CsrMatrix(pos, crd, val, (g * g, g * g), tune=True)
        s["d"] = (pos[1:] - pos[:-1]).to(torch.float64)
        s["mask"] = (torch.rand(g * g, generator=gen, device=DEV) >= 0.001).to(torch.float64)  # a few target nodes
    else:
        raise ValueError(op)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op in ("spmv_call", "pcg_call"):
        return s["fn"](*s["args"])
    if op == "spmv":
        return s["A"].spmv(s["x"], s["y"], accumulate=case["accumulate"])
    if op == "spmm":
        if case["format"] == "csr":
            return s["A"].spmm(s["B"], s["C"], accumulate=case["accumulate"])
        return device.spmm_dcsr(*s["A"], s["B"], s["C"], case["rows"])
    if op == "bspmm":
        return device.bspmm_csrv(*s["A"], s["B"], case["rows"])
    if op == "gemm":
        return device.bgemm(s["A"], s["B"], s["C"])
    if op == "pcg":
        return s["A"].pcg(s["b"], s["dinv"], 0.0, case["iters"])
    return s["A"].mht(s["mask"], s["d"], 0.95, 0.0, case["iters"])


def work(case):
    op, ib = case["op"], case.get("idx", 64) // 8
    if op in ("spmv_call", "spmv"):
        n = case["rows"]
        nnz = _grid_nnz(math.isqrt(n)) if case.get("dist") == "grid" else n * case["mean"]
        return {"bytes": nnz * (8 + ib) + (n + 1) * ib + 8 * n * (3 if case.get("accumulate", True) else 2), "flops": 2 * nnz}
    if op == "spmm":
        n, k = case["rows"], case["k"]
        nnz = n * case["mean"]
        reads_c = case["accumulate"] or case["format"] == "dcsr"
        lists = (2 if case["format"] == "dcsr" else 1) * (n + 1) * ib
        return {"bytes": nnz * (8 + ib) + lists + 8 * n * k * (3 if reads_c else 2), "flops": 2 * nnz * k}
    if op == "bspmm":
        n, e = case["rows"], case["nh"] * case["dh"]
        nnz = n * case["mean"]
        return {"bytes": nnz * (4 * case["nh"] + ib) + (n + 1) * ib + 8 * n * e, "flops": 2 * nnz * e}
    if op == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return {"bytes": 4 * b * (m * k + k * n + 2 * m * n), "flops": 2 * b * m * n * k}
    g = case["grid"]
    n = g * g
    if op == "mht":  # per iteration the matrix, mask and d, and x, r, p and the product read and written; two solves
        nnz, its, vectors = _grid_nnz(g, False), 2 * case["iters"], 10
    else:            # the same with dinv; a solve to a tolerance takes about 5 iterations per grid line
        nnz, its, vectors = _grid_nnz(g), case.get("iters", max(1, 5 * g // 2)), 9
    return {"bytes": its * (nnz * (8 + ib) + (n + 1) * ib + 8 * vectors * n), "flops": its * (2 * nnz + 12 * n)}


def tolerance(case):
    op = case["op"]
    if op == "gemm":
        return {"rel": 1e-5}   # fp32 sums
    if op == "bspmm":
        return {"rel": 1e-6}   # fp32 sums of a few dozen products
    if op in ("pcg", "pcg_call", "mht"):
        return {"rel": 1e-11}  # fp64; the order of a dot product's sum, amplified by the iterations
    return {"rel": 1e-14, "max": 1e-12}  # fp64 sums of up to 4096 products
