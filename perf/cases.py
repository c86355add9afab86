"""The work this package is measured on: whole sketch-preconditioned solves,
their differentiable form, and the products a caller makes on its own.

Every case is a plain dict; prepare() makes what a program holds before the
call (the matrix, the right-hand side, a workspace it keeps), run() makes one
pass through the public entry points, exact() the same outputs from plain
torch in FP64.  Matrices are A = G diag(c) with Gaussian G and column units c
spread over powers of ten, and solutions in the inverse units, so that every
column matters equally to b and an error of x is one number.
"""
import math

import torch

import tomos_b200 as tb
from tomos_b200.adjoint import lstsq

T = tb.TransposeType
ROWS = 1 << 17  # rows per block of the FP64 work

STORAGE = {"fp32": tb.NumericType.FP32, "fp16": tb.NumericType.FP16,
           "fp32_16": tb.NumericType.FP32_16, "fp32_bf16": tb.NumericType.FP32_BF16}
TIER = {"default": None, "accurate": tb.Tier.ACCURATE, "half": tb.Tier.HALF,
        "half_operands": tb.Tier.HALF_OPERANDS}


def listed():
    return [
        # Whole solves: CountSketch, sketch QR, preconditioned LSQR to a
        # backward error of 1e-6, through sketch_lsqr.
        # the smallest configuration: a solve is launches and latency
        _solve("solve_20000x200_fp32", 20000, 200, "fp32", noise=1e-6, decades=0.0),
        # the benchmark configuration, packed storage refined by exact passes
        _solve("solve_1000000x1000_fp32_16", 1000000, 1000, "fp32_16", noise=1e-8, decades=3.0),
        # a data matrix of any width: rows that start at any 4-byte address,
        # and a residual that does not vanish
        _solve("solve_150001x777_fp32", 150001, 777, "fp32", noise=1e-2, decades=1.0),
        # column-major, as a matrix file is read, packed
        _solve("solve_100000x300_col_fp32_16", 100000, 300, "fp32_16", layout="col", noise=1e-8, decades=2.0),
        # many rows, few columns: a regression on a long table
        _solve("solve_1000000x64_fp32_bf16", 1000000, 64, "fp32_bf16", noise=1e-2, decades=1.0),
        # sparse rows of ~20 entries, packed values
        _csr("solve_csr_500000x3000_fp32_16", "csr_solve", 500000, 3000, 20, "fp32_16"),
        # least squares inside a training step: 8 right-hand sides, forward
        # and the gradients of A and B
        {"name": "lstsq_200000x500x8", "kind": "lstsq", "m": 200000, "n": 500, "k": 8, "max_iters": 25},
        # The products on their own, each both ways (A x, then A^T u).
        # packed 16-bit tier of the benchmark matrix
        _mv("mv_1000000x1000_fp32_16", 1000000, 1000, "fp32_16", decades=3.0),
        # a small call of odd size: launch latency
        _mv("mv_2049x65_fp32", 2049, 65, "fp32", decades=1.0),
        # sparse rows, packed values read exactly
        _csr("mv_csr_2000000x5000_fp32_16", "csr_mv", 2000000, 5000, 20, "fp32_16", tier="accurate"),
        # 16 right-hand sides over one tall packed matrix, both ways
        _mm("mm_1000000x1000x16_fp32_16", "mm_tall", 1000000, 1000, 16, "fp32_16", "default"),
        # a square product on 16-bit operands
        _mm("mm_4096x4096x4096_fp32_16", "mm", 4096, 4096, 4096, "fp32_16", "half_operands"),
    ]


def _solve(name, m, n, storage, layout="row", noise=1e-8, decades=1.0):
    # Where b has a part outside range(A) the residual stalls at it and only
    # the pass that ends a cycle sees convergence: such a program keeps its
    # cycles short (the preconditioned iteration halves the error each step).
    return {"name": name, "kind": "solve", "m": m, "n": n, "storage": storage, "layout": layout,
            "noise": noise, "decades": decades, "max_iters": 25 if noise > 1e-3 else 200}


def _csr(name, kind, m, n, k, storage, tier="default"):
    return {"name": name, "kind": kind, "m": m, "n": n, "k": k, "storage": storage, "tier": tier, "max_iters": 200}


def _mv(name, m, n, storage, layout="row", tier="default", decades=1.0):
    return {"name": name, "kind": "mv", "m": m, "n": n, "storage": storage, "layout": layout, "tier": tier,
            "decades": decades}


def _mm(name, kind, m, n, k, storage, tier):
    return {"name": name, "kind": kind, "m": m, "n": n, "k": k, "storage": storage, "tier": tier}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "csr_solve", "lstsq", "mv", "mv", "csr_mv",
                       "mm_tall", "mm"])
    if kind == "solve":
        n = _log(rng, 32, 1000)
        m = _log(rng, max(5000, 20 * n), 1000000)
        storage = rng.choice(["fp32", "fp32_16", "fp32_bf16"])
        layout = rng.choice(["row", "row", "row", "col"])
        if layout == "col":
            m, n = min(m, 200000), min(n, 400)
        c = _solve(None, m, n, storage, layout, rng.choice([1e-8, 1e-6, 1e-2]), rng.choice([0.0, 1.0, 2.0]))
    elif kind == "csr_solve":
        n = _log(rng, 200, 3000)
        c = _csr(None, kind, _log(rng, max(50000, 20 * n), 500000), n, rng.randint(5, 30),
                 rng.choice(["fp32", "fp32_16"]))
    elif kind == "lstsq":
        n = _log(rng, 50, 500)
        c = {"kind": kind, "m": _log(rng, 20 * n, 200000), "n": n, "k": rng.randint(1, 8), "max_iters": 25}
    elif kind == "mv":
        m, n = _log(rng, 500, 1000000), _log(rng, 32, 1000)
        storage = rng.choice(["fp32", "fp16", "fp32_16", "fp32_bf16"])
        tier = rng.choice(["default", "accurate"]) if storage in ("fp32_16", "fp32_bf16") else "default"
        c = _mv(None, m, n, storage, rng.choice(["row", "row", "col"]), tier, rng.choice([0.0, 1.0, 2.0]))
    elif kind == "csr_mv":
        n = _log(rng, 200, 5000)
        c = _csr(None, kind, _log(rng, 20000, 2000000), n, rng.randint(5, 20), rng.choice(["fp32", "fp32_16"]),
                 "default")
    elif kind == "mm_tall":
        c = _mm(None, kind, _log(rng, 20000, 1000000), _log(rng, 64, 1000), rng.randint(2, 16),
                rng.choice(["fp32", "fp32_16"]), "default")
    else:
        storage = rng.choice(["fp32", "fp32_16", "fp32_bf16"])
        tier = "default" if storage == "fp32" else rng.choice(["default", "half", "half_operands"])
        c = _mm(None, kind, _log(rng, 256, 4096), _log(rng, 256, 4096), _log(rng, 256, 4096), storage, tier)
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _matrix(g, m, n, decades):
    """(A float32 m x n, column units c): A = G diag(c), c in 10^+-decades."""
    c = torch.pow(10.0, (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * decades)
    A = torch.randn(m, n, generator=g, device="cuda", dtype=torch.float32)
    A *= c.float()
    return A, c


def _product(A, x):
    """A x in FP64, row block by row block (A float32, x FP64 m x k)."""
    return torch.cat([A[r:r + ROWS].double() @ x for r in range(0, A.shape[0], ROWS)])


def _solve_inputs(case, seed):
    g = _gen(seed)
    m, n = case["m"], case["n"]
    A, c = _matrix(g, m, n, case["decades"])
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) / c
    b = _product(A, x[:, None])[:, 0]
    # noise relative to the size of b's entries
    b += case["noise"] * math.sqrt(n) * torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
    return A, b.float()


def _csr_inputs(case, seed):
    """k distinct uniform columns a row in increasing order, values with a
    row scale over 10^+-1 (rows of unequal weight), x, b with noise."""
    g = _gen(seed)
    m, n, k = case["m"], case["n"], case["k"]
    # k increasing distinct columns: sorted draws from n - k + 1 values, plus
    # their rank
    cols = torch.sort(torch.randint(0, n - k + 1, (m, k), generator=g, device="cuda"), dim=1).values
    cols = cols + torch.arange(k, device="cuda")
    scale = torch.pow(10.0, torch.rand(m, 1, generator=g, device="cuda", dtype=torch.float32) * 2 - 1)
    vals = torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32) * scale
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    b = (vals.double() * x[cols]).sum(1)
    b = b + 1e-8 * torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
    rp = torch.arange(0, (m + 1) * k, k, device="cuda", dtype=torch.int32)
    return rp, cols, vals, b.float(), g


def _store(A, storage, layout):
    """A user's Dense of this storage and layout from a float32 tensor."""
    m, n = A.shape
    if layout == "row":
        D = tb.Dense(tb.NumericType.FP32, tb.Layout.ROW_MAJOR, (m, n), n, A.reshape(-1))
    else:
        D = tb.Dense.from_tensor(A, tb.Layout.COL_MAJOR)
    return D if storage == "fp32" else tb.pack(D, STORAGE[storage])


def _store_csr(case, rp, cols, vals):
    flat = vals.reshape(-1).contiguous()
    if case["storage"] != "fp32":
        flat = tb.pack(tb.Dense.from_tensor(flat[None, :], tb.Layout.ROW_MAJOR), STORAGE[case["storage"]]).storage
    return tb.Csr(STORAGE[case["storage"]], (case["m"], case["n"]), rp,
                  cols.reshape(-1).to(torch.int32).contiguous(), flat)


def _rhs(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def prepare(case, seed):
    kind, m, n = case["kind"], case["m"], case["n"]
    st = dict(case)
    if kind == "solve":
        A, b = _solve_inputs(case, seed)
        st["A"], st["b"] = _store(A, case["storage"], case["layout"]), b
        st["ws"] = tb.create_lsqr_workspace(None, (m, n), tb.NumericType.FP32, tb.NumericType.FP64)
    elif kind == "csr_solve":
        rp, cols, vals, b, _ = _csr_inputs(case, seed)
        st["A"], st["b"] = _store_csr(case, rp, cols, vals), b
        st["ws"] = tb.create_lsqr_workspace(None, (m, n), tb.NumericType.FP32, tb.NumericType.FP64)
    elif kind == "lstsq":
        A, B, G = _lstsq_inputs(case, seed)
        st["A"], st["B"], st["G"] = A.requires_grad_(), B.requires_grad_(), G
    elif kind == "mv":
        g = _gen(seed)
        A, _ = _matrix(g, m, n, case["decades"])
        st["A"] = _store(A, case["storage"], case["layout"])
        st["x"], st["u"] = _rhs(g, n), _rhs(g, m)
        st["y"], st["z"] = torch.empty(m, device="cuda"), torch.empty(n, device="cuda")
    elif kind == "csr_mv":
        rp, cols, vals, _, g = _csr_inputs(case, seed)
        st["A"] = _store_csr(case, rp, cols, vals)
        st["x"], st["u"] = _rhs(g, n), _rhs(g, m)
        st["y"], st["z"] = torch.empty(m, device="cuda"), torch.empty(n, device="cuda")
    elif kind == "mm_tall":
        # row-major A; the right-hand sides column-major, as the vectors are
        A, B, U = _mm_tall_inputs(case, seed)
        st["A"] = _store(A, case["storage"], "row")
        st["B"], st["U"] = (tb.Dense.from_tensor(t, tb.Layout.COL_MAJOR) for t in (B, U))
        st["C"], st["D"] = (tb.Dense.create_strided(None, tb.Layout.COL_MAJOR, tb.NumericType.FP32, (r, case["k"]))
                            for r in (m, n))
    elif kind == "mm":
        A, B = _mm_inputs(case, seed)
        st["A"] = _store(A, case["storage"], "col")
        st["B"] = tb.Dense.from_tensor(B, tb.Layout.COL_MAJOR)
        st["C"] = tb.Dense.create_strided(None, tb.Layout.COL_MAJOR, tb.NumericType.FP32, (m, case["k"]))
    return st


def _lstsq_inputs(case, seed):
    g = _gen(seed)
    m, n, k = case["m"], case["n"], case["k"]
    A = _rhs(g, m, n)
    B = _product(A, _rhs(g, n, k).double()) + 1e-2 * math.sqrt(n) * _rhs(g, m, k).double()
    return A, B.float(), _rhs(g, n, k)


def _mm_tall_inputs(case, seed):
    g = _gen(seed)
    A, _ = _matrix(g, case["m"], case["n"], 1.0)
    return A, _rhs(g, case["n"], case["k"]), _rhs(g, case["m"], case["k"])


def _mm_inputs(case, seed):
    g = _gen(seed)
    return _rhs(g, case["m"], case["n"]), _rhs(g, case["n"], case["k"])


# ------------------------------------------------------------------ one pass

def run(st):
    kind = st["kind"]
    if kind in ("solve", "csr_solve"):
        x, _, d = tb.sketch_lsqr(st["A"], st["b"], 4 * st["n"], max_iters=st["max_iters"], workspace=st["ws"])
        return {"x": x, "d": d}
    if kind == "lstsq":
        X = lstsq(st["A"], st["B"], max_iters=st["max_iters"])
        gA, gB = torch.autograd.grad(X, (st["A"], st["B"]), st["G"])
        return {"X": X.detach(), "gA": gA, "gB": gB}
    tier = TIER[st["tier"]]
    if kind in ("mv", "csr_mv"):
        tb.mv_apply(tb.Device.CUDA, T.NO_TRANSPOSE, 1.0, st["A"], st["x"], 0.0, st["y"], tier=tier)
        tb.mv_apply(tb.Device.CUDA, T.TRANSPOSE, 1.0, st["A"], st["u"], 0.0, st["z"], tier=tier)
        return {"y": st["y"], "z": st["z"]}
    tb.mm_apply(tb.Device.CUDA, T.NO_TRANSPOSE, T.NO_TRANSPOSE, 1.0, st["A"], st["B"], 0.0, st["C"], tier=tier)
    if kind == "mm":
        return {"C": st["C"].view()}
    tb.mm_apply(tb.Device.CUDA, T.TRANSPOSE, T.NO_TRANSPOSE, 1.0, st["A"], st["U"], 0.0, st["D"], tier=tier)
    return {"C": st["C"].view(), "D": st["D"].view()}


# ------------------------------------------------------------------ what it needs

def _elem_bytes(case):
    if case["storage"] == "fp16":
        return 2
    two_byte = case["kind"] == "mm" and case["tier"] in ("half", "half_operands")
    two_byte = two_byte or (case["kind"] in ("mv", "csr_mv") and case["tier"] == "default"
                            and case["storage"] != "fp32")
    return 2 if two_byte else 4


def work(case):
    """Every input read once, every output written once; the flops of one
    product of each kind the result needs (a solve: the sketch, its QR and
    inverse, and one product pair)."""
    kind, m, n = case["kind"], case["m"], case["n"]
    qr = 2 * 4 * n * n * n - 2 * n ** 3 // 3 + n ** 3 // 3
    if kind == "solve":
        return {"bytes": 4 * m * n + 4 * m + 12 * n, "flops": qr + 6 * m * n}
    if kind == "csr_solve":
        z = m * case["k"]
        return {"bytes": 8 * z + 8 * m + 12 * n, "flops": qr + 6 * z}
    if kind == "lstsq":
        k = case["k"]  # A and B in, X, gA and gB out
        return {"bytes": 8 * m * n + 8 * m * k + 8 * n * k, "flops": qr + 2 * m * n + 10 * m * n * k}
    if kind == "mv":
        return {"bytes": _elem_bytes(case) * m * n + 8 * (m + n), "flops": 4 * m * n}
    if kind == "csr_mv":
        z = m * case["k"]
        return {"bytes": (4 + _elem_bytes(case)) * z + 4 * m + 8 * (m + n), "flops": 4 * z}
    k = case["k"]
    if kind == "mm_tall":
        return {"bytes": _elem_bytes(case) * m * n + 8 * (m + n) * k, "flops": 4 * m * n * k}
    return {"bytes": _elem_bytes(case) * m * n + 4 * n * k + 4 * m * k, "flops": 2 * m * n * k}


def tolerance(case):
    """About four times the distance from the FP64 result."""
    kind = case["kind"]
    if kind in ("solve", "csr_solve"):
        # a backward error below 1e-6 leaves 1e-5 to 5e-5 of x where the residual
        # vanishes; a cycle that runs its course leaves x's FP32 rounding and
        # the FP32 sums of 16-bit column norms d
        return {"rel": 2e-4 if case.get("noise", 0.0) < 1e-3 else 1e-5}
    if kind == "lstsq":
        return {"rel": 3e-5}  # the adjoint's products keep ~22 bits
    if kind in ("mv", "csr_mv"):
        return {"rel": 4e-7 if case["tier"] == "accurate" else 4e-6}  # FP32 sums
    return {"rel": 3e-5}  # FP32 sums over K of products to ~22 bits


# ------------------------------------------------------------------ FP64

def _half_only(A):
    """The 16-bit tier's value of float32 A stored as FP32_16: nine mantissa
    bits rounded to nearest even; below fp16's normal range a subnormal, by
    truncation of the ten-bit significand."""
    bits = A.view(torch.int32).to(torch.int64) & 0xFFFFFFFF
    e, mant = (bits >> 23) & 0xFF, bits & 0x7FFFFF
    hi, lo = mant >> 14, mant & 0x3FFF
    up = ((lo >> 13) & 1) & (((lo & 0x1FFF) != 0) | ((hi & 1) != 0)).to(torch.int64)
    hr = hi + up
    e = e + (hr >> 9)
    sig = 512 + (hr & 511)
    v = sig.double() * torch.pow(2.0, (e - 127 - 9).double())
    steps = (112 - e).clamp(0, 62)
    sub = (sig >> steps).double() * 2.0 ** -24
    v = torch.where(e >= 113, v, torch.where(e >= 99, sub, torch.zeros_like(v)))
    return torch.where(A < 0, -v, v)


def _decoded(A, storage, tier):
    """The FP64 values a product reads."""
    if storage == "fp16":
        return A.half().double()
    if storage == "fp32" or tier == "accurate":
        return A.double()
    if storage == "fp32_16":
        return _half_only(A)
    return (A.view(torch.int32) & -65536).view(torch.float32).double()


def _spd_solve(gram, rhs):
    """Solves gram x = rhs after scaling gram to a unit diagonal."""
    d = gram.diagonal().sqrt()
    L = torch.linalg.cholesky(gram / d[:, None] / d[None, :])
    rhs = rhs / d[:, None]
    return torch.cholesky_solve(rhs, L) / d[:, None]


def exact(case, seed):
    kind, m, n = case["kind"], case["m"], case["n"]
    if kind == "solve":
        A, b = _solve_inputs(case, seed)
        gram = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        rhs = torch.zeros(n, 1, device="cuda", dtype=torch.float64)
        for r in range(0, m, ROWS):
            blk = A[r:r + ROWS].double()
            gram += blk.T @ blk
            rhs += blk.T @ b[r:r + ROWS].double()[:, None]
        # a step of refinement from the FP64 residual
        x = _spd_solve(gram, rhs)
        res = b.double()[:, None] - _product(A, x)
        g = sum(A[r:r + ROWS].double().T @ res[r:r + ROWS] for r in range(0, m, ROWS))
        x = x + _spd_solve(gram, g)
        # the column norms of the values the sketch reads (16 bits of packed A)
        cs = sum(_decoded(A[r:r + ROWS], case["storage"], "default").square().sum(0) for r in range(0, m, ROWS))
        return {"x": x[:, 0], "d": cs.sqrt()}
    if kind == "csr_solve":
        _, cols, vals, b, _ = _csr_inputs(case, seed)
        gram = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        rhs = torch.zeros(n, 1, device="cuda", dtype=torch.float64)
        for r in range(0, m, ROWS // 4):
            c, v = cols[r:r + ROWS // 4], vals[r:r + ROWS // 4].double()
            blk = torch.zeros(c.shape[0], n, device="cuda", dtype=torch.float64).scatter_(1, c, v)
            gram += blk.T @ blk
            rhs += blk.T @ b[r:r + ROWS // 4].double()[:, None]
        v = _decoded(vals, case["storage"], "default")
        cs = torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, cols.reshape(-1),
                                                                           v.square().reshape(-1))
        return {"x": _spd_solve(gram, rhs)[:, 0], "d": cs.sqrt()}
    if kind == "lstsq":
        A, B, G = _lstsq_inputs(case, seed)
        A, B, G = A.double(), B.double(), G.double()
        gram = A.T @ A
        X = _spd_solve(gram, A.T @ B)
        X = X + _spd_solve(gram, A.T @ (B - A @ X))
        lam = _spd_solve(gram, G)
        gB = A @ lam
        return {"X": X, "gA": (B - A @ X) @ lam.T - gB @ X.T, "gB": gB}
    if kind == "mv":
        g = _gen(seed)
        A, _ = _matrix(g, m, n, case["decades"])
        x, u = _rhs(g, n).double(), _rhs(g, m).double()
        y, z = [], torch.zeros(n, device="cuda", dtype=torch.float64)
        for r in range(0, m, ROWS):
            blk = _decoded(A[r:r + ROWS], case["storage"], case["tier"])
            y.append(blk @ x)
            z += blk.T @ u[r:r + ROWS]
        return {"y": torch.cat(y), "z": z}
    if kind == "csr_mv":
        _, cols, vals, _, g = _csr_inputs(case, seed)
        x, u = _rhs(g, n).double(), _rhs(g, m).double()
        v = _decoded(vals, case["storage"], case["tier"])
        z = torch.zeros(n, device="cuda", dtype=torch.float64)
        z.index_add_(0, cols.reshape(-1), (v * u[:, None]).reshape(-1))
        return {"y": (v * x[cols]).sum(1), "z": z}
    if kind == "mm_tall":
        A, B, U = _mm_tall_inputs(case, seed)
        D = sum(A[r:r + ROWS].double().T @ U[r:r + ROWS].double() for r in range(0, m, ROWS))
        return {"C": _product(A, B.double()), "D": D}
    A, B = _mm_inputs(case, seed)
    tier = case["tier"]
    if tier == "half_operands":
        B = B.half() if case["storage"] == "fp32_16" else B.bfloat16()
    tier = "accurate" if tier == "default" else "default"
    return {"C": _decoded(A, case["storage"], tier) @ B.double()}
