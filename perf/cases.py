"""The calls whose time matters to a user of ozblas_b200, each through the package's public entry points.

listed() names them, draw() gives more of the same ranges, prepare() makes what a program holds before the call
(device inputs with the harness's phi distribution, (U(0,1) - 0.5) exp(phi N(0,1)), output buffers and a handle),
run() is one call, work() the bytes and operations of its result, exact() the result in plain 64-bit torch.
"""
import math

import torch

import ozblas_b200 as ozb

WORK_BYTES = 8 << 30  # the handle's arena, as the benchmark's


def listed():
    return [
        # A reproducible dot product of a short vector: an inner call of a solver, all latency and launches.
        {"name": "ddot_small", "kind": "ddot", "n": 1000, "phi": 1.0, "sum": 0},
        # The benchmark's DOT: 2^24 elements in the default ordered sum.
        {"name": "ddot_2p24", "kind": "ddot", "n": 1 << 24, "phi": 2.0, "sum": 0},
        # A correctly rounded norm of an odd-length vector that fits L2.
        {"name": "dnrm2_5m", "kind": "dnrm2", "n": 5000001, "phi": 2.0, "sum": 1},
        # The benchmark's GEMV: y = A x, 8192 x 8192.
        {"name": "dgemv_n_8192", "kind": "dgemv", "trans": "n", "m": 8192, "n": 8192, "phi": 1.0, "sum": 0},
        # y = A^T x with odd sizes: the other direction of a least-squares or bi-orthogonal iteration.
        {"name": "dgemv_t_odd", "kind": "dgemv", "trans": "t", "m": 6001, "n": 3001, "phi": 1.0, "sum": 0},
        # The benchmark's sparse product: the 7-point stencil on 128^3.
        {"name": "dcsrmv_128", "kind": "dcsrmv", "gx": 128, "gy": 128, "gz": 128, "rows": "stencil", "phi": 1.0, "sum": 0},
        # A reproducible conjugate-gradient solve on the benchmark's 100^3 Poisson problem, first 100 iterations.
        {"name": "dcg_100", "kind": "dcg", "gx": 100, "gy": 100, "gz": 100, "iters": 100, "sum": 1},
        # The plain FP64-slice GEMM, 1024^3: the bit-reproducible product at the size of the parity benchmark.
        {"name": "dgemm_1024", "kind": "dgemm", "ta": "n", "tb": "n", "m": 1024, "n": 1024, "k": 1024, "phi": 1.0,
         "sum": 0, "fast": 0, "alpha": 1.0, "beta": 0.0},
        # The same form on ragged sizes with a transpose and an update of C.
        {"name": "dgemm_ragged", "kind": "dgemm", "ta": "t", "tb": "n", "m": 3001, "n": 1999, "k": 2500, "phi": 1.0,
         "sum": 0, "fast": 0, "alpha": 1.5, "beta": -0.5},
        # The headline: INT8 precision form at 8192^3, triangular pair set.
        {"name": "dgemm_i8_8192", "kind": "dgemm_i8", "ta": "n", "tb": "n", "m": 8192, "n": 8192, "k": 8192,
         "phi": 1.0, "fast": 1, "alpha": 1.0, "beta": 0.0},
        # 256 uneven INT8 products in one grouped call, full pair sets.
        {"name": "dgemm_i8_batched", "kind": "batched", "count": 256, "shapes": 5, "fast": 0},
        # Single-precision data with reproducible results (FP64 slices), 2048^3.
        {"name": "sdgemm_2048", "kind": "sdgemm", "ta": "n", "tb": "n", "m": 2048, "n": 2048, "k": 2048, "phi": 1.0,
         "fast": 0, "alpha": 1.0, "beta": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mnk(rng, lo, hi, cap):
    while True:
        m, n, k = (_log(rng, lo, hi) for _ in range(3))
        if m * n * k <= cap ** 3:
            return m, n, k


def draw(rng):
    kind = rng.choice(["ddot", "dnrm2", "dgemv", "dcsrmv", "dcg", "dgemm", "dgemm_i8", "batched", "dsgemm", "sdgemm",
                       "qgemm"])
    phi, s = rng.choice([0.5, 1.0, 2.0]), rng.choice([0, 1])
    if kind in ("ddot", "dnrm2"):
        return {"kind": kind, "n": _log(rng, 100, 1 << 24), "phi": phi, "sum": s}
    if kind == "dgemv":
        return {"kind": kind, "trans": rng.choice("nt"), "m": _log(rng, 64, 8192), "n": _log(rng, 64, 8192),
                "phi": phi, "sum": s}
    if kind == "dcsrmv":
        return {"kind": kind, "gx": _log(rng, 10, 128), "gy": _log(rng, 10, 128), "gz": _log(rng, 10, 128),
                "rows": rng.choice(["stencil", "random"]), "phi": phi, "sum": s}
    if kind == "dcg":
        return {"kind": kind, "gx": _log(rng, 10, 100), "gy": _log(rng, 10, 100), "gz": _log(rng, 10, 100),
                "iters": _log(rng, 10, 100), "sum": s}
    if kind == "batched":
        return {"kind": kind, "count": _log(rng, 4, 200), "shapes": rng.randrange(1 << 20), "fast": rng.choice([0, 1])}
    case = {"kind": kind, "ta": rng.choice("nt"), "tb": rng.choice("nt"), "phi": phi,
            "fast": rng.choice([0, 1]), "alpha": rng.choice([1.0, 1.5]), "beta": rng.choice([0.0, -0.5])}
    if kind == "dgemm_i8":
        case["phi"] = rng.choice([0.5, 1.0, 2.0, 4.0])
        m, n, k = _mnk(rng, 64, 8192, 5000)
    elif kind == "dgemm":
        case["sum"] = s
        m, n, k = _mnk(rng, 64, 4096, 2500)
    elif kind == "qgemm":
        m, n, k = _mnk(rng, 64, 2048, 1024)
    else:
        m, n, k = _mnk(rng, 64, 4096, 2048)
    return {**case, "m": m, "n": n, "k": k}


def _phi(gen, shape, phi, dtype=torch.float64):
    u = torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)
    z = torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    return u.sub_(0.5).mul_(z.mul_(phi).exp_()).to(dtype)


def _shapes(case):
    """The batch's (m, n, k) triples, log-uniform in [64, 2048], and each problem's phi."""
    g = torch.Generator().manual_seed(case["shapes"])
    u = torch.rand((case["count"], 4), dtype=torch.float64, generator=g).tolist()
    lo, hi = math.log(64), math.log(2048)
    return [tuple(int(math.exp(lo + (hi - lo) * v)) for v in r[:3]) for r in u], [(0.5, 1.0, 2.0, 4.0)[int(4 * r[3])] for r in u]


def _csr(case, gen):
    """(rowptr, colind, grid size): the 7-point stencil in natural order, or rows of 1 to 12 random columns."""
    gx, gy, gz = case["gx"], case["gy"], case["gz"]
    m = gx * gy * gz
    i = torch.arange(m, dtype=torch.int64, device="cuda")
    if case.get("rows", "stencil") == "random":
        ln = torch.randint(1, 13, (m,), device="cuda", generator=gen)
        rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
        rowptr[1:] = torch.cumsum(ln, 0)
        col = torch.randint(0, m, (int(rowptr[-1]),), device="cuda", generator=gen)
        return rowptr.to(torch.int32), col.to(torch.int32), None
    x, y, z = i % gx, (i // gx) % gy, i // (gx * gy)
    near = [(-gx * gy, z > 0), (-gx, y > 0), (-1, x > 0), (0, x >= 0), (1, x < gx - 1), (gx, y < gy - 1),
            (gx * gy, z < gz - 1)]
    col = torch.stack([i + o for o, _ in near], 1)
    has = torch.stack([k for _, k in near], 1)
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(has.sum(1), 0)
    return rowptr.to(torch.int32), col[has].to(torch.int32), has


def _quad(a, gen):
    """Binary128 values with a's sign, exponent and fraction and 60 random low bits: int64 pairs (lo, hi)."""
    bits = a.view(torch.int64)
    low = torch.randint(0, 1 << 60, a.shape, device="cuda", generator=gen)
    frac = bits & ((1 << 52) - 1)
    hi = (bits & (-1 << 63)) | ((((bits >> 52) & 0x7FF) + 15360) << 48) | (frac >> 4)
    return torch.stack([((frac & 15) << 60) | low, hi], dim=-1).contiguous()


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, d = case["kind"], {}
    if kind in ("ddot", "dnrm2"):
        d["x"] = _phi(gen, (case["n"],), case["phi"])
        if kind == "ddot":
            d["y"] = _phi(gen, (case["n"],), case["phi"])
    elif kind == "dgemv":  # A is m x n column-major: the tensor holds its n columns as rows
        d["A"] = _phi(gen, (case["n"], case["m"]), case["phi"])
        d["x"] = _phi(gen, (case["n"] if case["trans"] == "n" else case["m"],), case["phi"])
    elif kind in ("dcsrmv", "dcg"):
        d["rowptr"], d["colind"], has = _csr(case, gen)
        m = d["rowptr"].numel() - 1
        if kind == "dcsrmv":
            d["val"] = _phi(gen, (d["colind"].numel(),), case["phi"])
            d["x"] = _phi(gen, (m,), case["phi"])
        else:
            V = torch.full((m, 7), -1.0, dtype=torch.float64, device="cuda")
            V[:, 3] = 6.0 + 0.01 * torch.rand(m, dtype=torch.float64, device="cuda", generator=gen)
            d["val"] = V[has]
            near = torch.zeros((m, 7), dtype=torch.int64, device="cuda")
            near[has] = d["colind"].long()
            xt = torch.randn(m, dtype=torch.float64, device="cuda", generator=gen)
            d["b"] = (V * has * xt[near]).sum(1)  # A x_true, in a fixed order
    elif kind == "batched":
        shapes, phis = _shapes(case)
        d["A"] = [_phi(gen, (k, m), p) for (m, n, k), p in zip(shapes, phis)]
        d["B"] = [_phi(gen, (n, k), p) for (m, n, k), p in zip(shapes, phis)]
    else:
        m, n, k = case["m"], case["n"], case["k"]
        dtype = torch.float32 if kind == "sdgemm" else torch.float64
        d["A"] = _phi(gen, (k, m) if case["ta"] == "n" else (m, k), case["phi"], dtype)
        d["B"] = _phi(gen, (n, k) if case["tb"] == "n" else (k, n), case["phi"], dtype)
        d["C0"] = _phi(gen, (n, m), 1.0, dtype)
        if kind == "qgemm":
            d = {key: _quad(v, gen) for key, v in d.items()}
    return d


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    kind = case["kind"]
    h = s["h"] = ozb.Handle(WORK_BYTES, stream=torch.cuda.current_stream())
    h.sumMode, h.fastMode = case.get("sum", 0), case.get("fast", 0)
    f64 = {"dtype": torch.float64, "device": "cuda"}
    if kind == "dgemv":
        s["y"] = torch.zeros(case["m"] if case["trans"] == "n" else case["n"], **f64)
    elif kind == "dcsrmv":
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "dcg":
        s["x"] = torch.zeros_like(s["b"])
    elif kind == "batched":
        shapes, _ = _shapes(case)
        s["ms"], s["ns"], s["ks"] = (list(v) for v in zip(*shapes))
        s["out"] = torch.zeros(sum(m * n for m, n, _ in shapes), **f64)
        s["C"] = list(torch.split(s["out"], [m * n for m, n, _ in shapes]))
        s["one"], s["zero"] = [1.0] * len(shapes), [0.0] * len(shapes)
    elif "C0" in s:
        s["C"] = s["C0"].clone()
        if kind == "qgemm":
            q = {0.0: (0, 0), 1.0: (0, 0x3FFF << 48), 1.5: (0, 0x3FFF8 << 44), -0.5: (0, 0xBFFE << 48)}
            s["alpha"], s["beta"] = q[case["alpha"]], q[case["beta"]]
        else:
            s["alpha"], s["beta"] = case["alpha"], case["beta"]
    return s


def run(s):
    c, h = s["case"], s["h"]
    kind = c["kind"]
    if kind == "ddot":
        return ozb.ddot(h, c["n"], s["x"], s["y"])
    if kind == "dnrm2":
        return ozb.dnrm2(h, c["n"], s["x"])
    if kind == "dgemv":
        ozb.dgemv(h, c["trans"], c["m"], c["n"], 1.0, s["A"], c["m"], s["x"], 0.0, s["y"])
        return s["y"]
    if kind == "dcsrmv":
        m = s["y"].numel()
        ozb.dcsrmv(h, "n", m, m, s["val"].numel(), 1.0, s["val"], s["colind"], s["rowptr"], s["x"], 0.0, s["y"])
        return s["y"]
    if kind == "dcg":
        s["x"].zero_()
        m = s["b"].numel()
        its = ozb.dcg(h, "n", m, s["val"].numel(), s["val"], s["colind"], s["rowptr"], s["b"], s["x"], c["iters"], 0.0)
        return {"x": s["x"], "iterations": its}
    if kind == "batched":
        ozb.dgemm_i8_batched(h, "n", "n", s["ms"], s["ns"], s["ks"], s["one"], s["A"], s["ms"], s["B"], s["ks"],
                             s["zero"], s["C"], s["ms"])
        return s["out"]
    m, n, k = c["m"], c["n"], c["k"]
    if c["beta"] != 0.0:
        s["C"].copy_(s["C0"])
    call = {"dgemm": ozb.dgemm, "dgemm_i8": ozb.dgemm_i8, "dsgemm": ozb.dsgemm, "sdgemm": ozb.sdgemm, "qgemm": ozb.qgemm}
    call[kind](h, c["ta"], c["tb"], m, n, k, s["alpha"], s["A"], m if c["ta"] == "n" else k, s["B"],
               k if c["tb"] == "n" else n, s["beta"], s["C"], m)
    return s["C"]


def work(case):
    kind = case["kind"]
    if kind in ("ddot", "dnrm2"):
        n = case["n"]
        return {"bytes": (16 if kind == "ddot" else 8) * n, "flops": 2 * n}
    if kind == "dgemv":
        m, n = case["m"], case["n"]
        return {"bytes": 8 * (m * n + m + n), "flops": 2 * m * n}
    if kind in ("dcsrmv", "dcg"):
        gx, gy, gz = case["gx"], case["gy"], case["gz"]
        m = gx * gy * gz
        nnz = 7 * m - 2 * (gx * gy + gy * gz + gx * gz) if case.get("rows", "stencil") == "stencil" else int(6.5 * m)
        one = 12 * nnz + 4 * (m + 1) + 16 * m
        if kind == "dcsrmv":
            return {"bytes": one, "flops": 2 * nnz}
        # an iteration: the product, <p, q>, the updates of x and r with <r, r>, the update of p
        return {"bytes": case["iters"] * (one + 72 * m), "flops": case["iters"] * (2 * nnz + 10 * m)}
    if kind == "batched":
        shapes, _ = _shapes(case)
        return {"bytes": sum(8 * (m * k + k * n + m * n) for m, n, k in shapes),
                "flops": sum(2 * m * n * k for m, n, k in shapes)}
    m, n, k = case["m"], case["n"], case["k"]
    size = {"sdgemm": 4, "qgemm": 16}.get(kind, 8)
    return {"bytes": size * (m * k + k * n + m * n * (2 if case["beta"] != 0.0 else 1)), "flops": 2 * m * n * k}


def _spmv(d, v):
    rows = torch.repeat_interleave(torch.arange(d["rowptr"].numel() - 1, device="cuda"), (d["rowptr"][1:] - d["rowptr"][:-1]).long())
    y = torch.zeros(d["rowptr"].numel() - 1, dtype=torch.float64, device="cuda")
    return y.index_add_(0, rows, d["val"] * v[d["colind"].long()])


def exact(case, seed):
    kind = case["kind"]
    if kind == "qgemm":  # binary128 results as bit pairs
        return None
    d = _inputs(case, seed)
    if kind == "ddot":
        return float((d["x"] * d["y"]).sum())
    if kind == "dnrm2":
        return math.sqrt(float((d["x"] * d["x"]).sum()))
    if kind == "dgemv":
        return (d["A"].t() if case["trans"] == "n" else d["A"]) @ d["x"]
    if kind == "dcsrmv":
        return _spmv(d, d["x"])
    if kind == "dcg":
        x = torch.zeros_like(d["b"])
        r = d["b"].clone()
        p, old = r.clone(), r @ r
        for _ in range(case["iters"]):
            q = _spmv(d, p)
            a = old / (p @ q)
            x, r = x + a * p, r - a * q
            new = r @ r
            p, old = r + (new / old) * p, new
        return {"x": x, "iterations": None}
    if kind == "batched":
        return torch.cat([(B @ A).reshape(-1) for A, B in zip(d["A"], d["B"])])
    A, B, C = d["A"].double(), d["B"].double(), d["C0"].double()
    opA, opB = A if case["ta"] == "n" else A.t(), B if case["tb"] == "n" else B.t()
    return case["alpha"] * (opB @ opA) + (case["beta"] * C if case["beta"] != 0.0 else 0.0)
