"""The work a program gives this library, for timing it: whole solves of
y = exp(tA)v through the public Python entry points, from the smallest
problem of the tests to the full-size ones of the benchmark, in each
precision, step controller and orthogonalisation form, and batches.

A context holds the matrix (and its basis) as a program keeps it between
solves; a solve takes a start vector and returns y. The FP64 forms return y
in FP64 with the accept/reject counts; the mixed forms, whose results are
good to about FP32's precision (relative errors of 1e-7), hand y on in FP32.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "matrix-exp-krylov_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

from mexk.api import Context  # noqa: E402
from mexk.batch import Batch  # noqa: E402
from mexk.synthetic import CSR  # noqa: E402

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def solve(name, matrix, size, t, m, **kw):
    case = {"name": name, "kind": "solve", "matrix": matrix, "size": size, "pe": 0.0, "degree": 0, "t": t, "m": m,
            "m_alloc": m, "tol": 1e-6, "max_restarts": 0, "precision": "fp64", "controller": "reference",
            "window": 0, "host": False}
    case.update(kw)
    return case


def batch(name, problems, rows_lo, rows_hi, m):
    return {"name": name, "kind": "batch", "problems": problems, "rows_lo": rows_lo, "rows_hi": rows_hi, "m": m,
            "tol": 1e-6}


def heat_t(N):
    """A time with t|A| as the full-size heat workload's (t = 1e-5 at N = 2048)."""
    return 1e-5 * (2049.0 / (N + 1)) ** 2


def listed():
    return [
        # The plain method on the small random matrix, host vectors: what a program written
        # for the reference's ArnoldiRunner calls (latency and launches count).
        solve("random_2000_fp64_host", "random", 2000, 1.0, 30, degree=10, host=True),
        # The same matrix in mixed precision with the candidate-step search, device vectors.
        solve("random_2000_mixed_search", "random", 2000, 1.0, 30, degree=10, precision="mixed", controller="search"),
        # The reference's ArnoldiParams defaults (m = 100, tol 1e-8, 10 restarts) on an ordinary random matrix.
        solve("random_50021_fp64_defaults", "random", 50021, 1.0, 100, degree=10, tol=1e-8, max_restarts=10),
        # A small heat grid, plain method: many short cycles with rejects (the CLI's settings).
        solve("heat_96_fp64", "heat", 96, heat_t(96), 30),
        # The full-size heat equation, plain method: the form every other one is held to.
        solve("heat_2048_fp64", "heat", 2048, 1e-5, 30),
        # The same in the form the benchmark chooses: mixed, learned controller, window 2.
        solve("heat_2048_mixed_learned_w2", "heat", 2048, 1e-5, 30, m_alloc=60, precision="mixed",
              controller="learned", window=2),
        # An odd grid of ordinary size, FP64 short recurrence with the search.
        solve("heat_777_fp64_search_w2", "heat", 777, heat_t(777), 30, controller="search", window=2),
        # Irregular rows (Zipf lengths, scattered columns): full Arnoldi in mixed precision, a large one.
        solve("powerlaw_2097152_mixed_search", "powerlaw", 2097152, 0.5, 40, precision="mixed", controller="search"),
        # The same kind in plain FP64, an odd ordinary size.
        solve("powerlaw_300007_fp64", "powerlaw", 300007, 0.5, 40),
        # 3D convection-diffusion at the benchmark's size with the learned controller.
        solve("convdiff_128_mixed_learned", "convdiff", 128, 1e-3, 30, pe=100.0, m_alloc=60, precision="mixed",
              controller="learned"),
        # The same operator on an odd grid, plain method.
        solve("convdiff_61_fp64", "convdiff", 61, 1e-3, 30, pe=10.0),
        # A batch of uneven random problems with 16 start vectors each, results fetched.
        batch("batch_12_uneven", 12, 10000, 60000, 30),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def form(symmetric, m):
        """(precision, controller, window, m_alloc) as programs combine them."""
        precision = rng.choice(["fp64", "mixed"])
        controller = rng.choice(["reference", "search"] if precision == "fp64" else ["search", "learned"])
        window = 2 if symmetric and rng.random() < 0.5 else 0
        return {"precision": precision, "controller": controller, "window": window,
                "m_alloc": 60 if controller == "learned" else m}

    kind = rng.choice(["random", "heat", "powerlaw", "convdiff", "defaults", "batch"])
    if kind == "random":
        m = rng.choice([20, 30, 40])
        case = solve("", "random", log(1500, 400000), rng.uniform(0.3, 1.5), m, degree=rng.randint(5, 20),
                     **form(False, m))
        case["host"] = case["size"] < 5000 and rng.random() < 0.5
    elif kind == "defaults":
        case = solve("", "random", log(1500, 100000), rng.uniform(0.5, 1.0), rng.choice([80, 100, 128]),
                     degree=rng.randint(5, 20), tol=1e-8, max_restarts=10)
        case["m_alloc"] = case["m"]
    elif kind == "heat":
        N = log(48, 1500)
        m = rng.choice([20, 30, 40])
        case = solve("", "heat", N, heat_t(N) * rng.uniform(0.2, 1.0), m, **form(True, m))
    elif kind == "powerlaw":
        m = rng.choice([30, 40])
        case = solve("", "powerlaw", log(2048, 1500000), rng.uniform(0.2, 0.5), m, **form(False, m))
        if case["precision"] == "fp64":
            case["size"] = min(case["size"], 300000 + rng.randint(0, 99))
    elif kind == "convdiff":
        N = log(14, 110)
        m = rng.choice([20, 30, 40])
        case = solve("", "convdiff", N, 1e-3 * rng.uniform(0.3, 1.0) * min(4.0, (129.0 / (N + 1)) ** 2), m,
                     pe=rng.choice([1.0, 10.0, 100.0]), **form(False, m))
    else:
        lo = log(1000, 20000)
        case = batch("", rng.randint(2, 12), lo, lo * rng.randint(2, 3), rng.choice([16, 24, 30]))
    del case["name"]
    return case


# ------------------------------------------------------------------ matrices
def stencil(shape, offsets, values):
    """CSR of a Dirichlet stencil on a grid (axis 0 fastest): at each point,
    values[q] times the neighbour offsets[q] (ascending column order)."""
    n = math.prod(shape)
    p = torch.arange(n, device=DEV)
    at, rest = [], p
    for s in shape:
        at.append(rest % s)
        rest = rest // s
    cols, ok = [], []
    for off in offsets:
        c, inside, step = p, torch.ones_like(p, dtype=torch.bool), 1
        for a, o, s in zip(at, off, shape):
            c = c + o * step
            inside = inside & (a + o >= 0) & (a + o < s)
            step *= s
        cols.append(c)
        ok.append(inside)
    ok = torch.stack(ok, 1)
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row_ptr[1:] = ok.sum(1).cumsum(0)
    vals = torch.tensor(values, dtype=torch.float64, device=DEV).expand(n, -1)
    return CSR(n, row_ptr.to(torch.int32).cpu().numpy(), torch.stack(cols, 1)[ok].to(torch.int32).cpu().numpy(),
               vals[ok].cpu().numpy())


@functools.lru_cache(maxsize=2)
def heat_matrix(N):
    inv = float((N + 1) ** 2)
    return stencil((N, N), [(0, -1), (-1, 0), (0, 0), (1, 0), (0, 1)], [inv, inv, -4.0 * inv, inv, inv])


@functools.lru_cache(maxsize=2)
def convdiff_matrix(N, pe):
    back, diag, fwd = zip(*(convdiff_axis(N, pe, d) for d in range(3)))
    offsets = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    return stencil((N, N, N), offsets, [back[2], back[1], back[0], sum(diag), fwd[0], fwd[1], fwd[2]])


def convdiff_axis(N, pe, d):
    """(backward, diagonal, forward) entries of the operator along axis d."""
    inv2, b = float((N + 1) ** 2), (1.0, 0.5, 0.25)[d] * pe * (N + 1)
    return inv2 + b, -2.0 * inv2 - b, inv2


def scattered_csr(n, degrees, scale, shift, gen):
    """Rows with about degrees[i] uniform off-diagonal columns, values uniform
    on a grid of 2^-20 in [-scale, scale], diagonal -(row |off| sum) - shift
    (exact in FP64: the same matrix on every run)."""
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), degrees)
    cols = torch.randint(0, n - 1, (rows.numel(),), generator=gen, device=DEV)
    cols += (cols >= rows).to(cols.dtype)
    off = torch.unique(rows * n + cols)  # sorted; a column drawn twice counts once
    v = torch.randint(-(1 << 20), (1 << 20) + 1, (off.numel(),), generator=gen, device=DEV).double() / (1 << 20) * scale
    r = off // n
    diag = torch.full((n,), -shift, dtype=torch.float64, device=DEV).index_add_(0, r, -v.abs())
    i = torch.arange(n, device=DEV)
    key, order = torch.sort(torch.cat([off, i * n + i]))
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row_ptr[1:] = (torch.bincount(r, minlength=n) + 1).cumsum(0)
    return CSR(n, row_ptr.to(torch.int32).cpu().numpy(), (key % n).to(torch.int32).cpu().numpy(),
               torch.cat([v, diag])[order].cpu().numpy())


def random_matrix(n, degree, gen):
    return scattered_csr(n, torch.full((n,), degree, device=DEV), 0.5, 1.0, gen)


def powerlaw_matrix(n, gen):
    """Off-diagonal counts Zipf (s = 1.8) clipped to [2, 2048]."""
    # P(k) by the partial sums of k^-1.8; the tail past 2048 is clipped to it
    k = np.arange(1, 2048, dtype=np.float64)
    zeta = 1.882229618102822  # sum of k^-1.8 over all k
    cdf = torch.from_numpy(np.cumsum(k ** -1.8) / zeta).to(DEV)
    u = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    deg = (torch.searchsorted(cdf, u) + 1).clamp(2, min(2048, n - 1))
    return scattered_csr(n, deg, 1.0, 0.5, gen)


def generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def make_matrix(case, gen):
    if case["matrix"] == "heat":
        return heat_matrix(case["size"])
    if case["matrix"] == "convdiff":
        return convdiff_matrix(case["size"], case["pe"])
    if case["matrix"] == "powerlaw":
        return powerlaw_matrix(case["size"], gen)
    return random_matrix(case["size"], case["degree"], gen)


def start_vector(case, n, gen):
    if case["matrix"] in ("heat", "convdiff"):
        return torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    return torch.randn(n, generator=gen, device=DEV, dtype=torch.float64)


def batch_problems(case, seed):
    """(A, V (16, rows), t) of each problem: rows spread evenly over the
    logarithm of the case's range, degrees over 5..20, the rest from the seed."""
    gen = generator(seed)
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["problems"]):
        n = int(round(case["rows_lo"] * (case["rows_hi"] / case["rows_lo"]) ** ((i + 0.5) / case["problems"])))
        A = random_matrix(n, 5 + 7 * i % 16, gen)
        V = torch.randn((16, n), generator=gen, device=DEV, dtype=torch.float64)
        out.append((A, V, float(rng.uniform(0.1, 2.0))))
    return out


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    if case["kind"] == "batch":
        b = Batch(m=case["m"], tol=case["tol"])
        probs = batch_problems(case, seed)
        for A, V, t in probs:
            b.add(A, V.cpu().numpy(), t)
        b.upload()
        return {"batch": b, "count": len(probs)}
    gen = generator(seed)
    A = make_matrix(case, gen)
    ctx = Context(A, m_alloc=case["m_alloc"])
    v = start_vector(case, A.n, gen)
    args = {"t": case["t"], "m": case["m"], "tol": case["tol"], "max_restarts": case["max_restarts"],
            "precision": case["precision"], "controller": case["controller"], "window": case["window"]}
    if case["host"]:
        return {"ctx": ctx, "v": v.cpu().numpy(), "args": args, "host": True}
    return {"ctx": ctx, "v": v, "y": torch.empty_like(v), "args": args, "host": False}


def run(state):
    if "batch" in state:
        b = state["batch"]
        b.run()
        return [b.result(i)[0].astype(np.float32) for i in range(state["count"])]
    args = state["args"]
    if state["host"]:
        y, res = state["ctx"].expmv(state["v"], **args)
    else:
        y = state["y"]
        res = state["ctx"].expmv_device(state["v"].data_ptr(), y.data_ptr(), **args)
    if args["precision"] == "mixed":
        return y.astype(np.float32) if state["host"] else y.float()
    return {"y": y, "accepted": res["restarts_done"], "attempts": res["attempts"]}


def work(case):
    """The matrix (4-byte indices, values of the precision) and v read once, y
    written once; the arithmetic of one basis of m columns: its products and
    its two-pass orthogonalisation (against the window's columns)."""
    if case["kind"] == "batch":
        n = case["problems"] * math.sqrt(case["rows_lo"] * case["rows_hi"])
        nnz, value, m, rhs = 13.5 * n, 4, case["m"], 16
        columns = m * (m + 1) / 2
    else:
        s = case["size"]
        n = {"heat": s ** 2, "convdiff": s ** 3}.get(case["matrix"], s)
        per = {"heat": 5.0, "convdiff": 7.0, "powerlaw": 14.5}.get(case["matrix"], case["degree"] + 1.0)
        nnz, value, m, rhs = per * n, 4 if case["precision"] == "mixed" else 8, case["m"], 1
        columns = 2 * m - 1 if case["window"] else m * (m + 1) / 2
    return {"bytes": nnz * (4 + value) + 4 * n + 16 * n * rhs, "flops": rhs * (2 * nnz * m + 8 * n * columns)}


# ------------------------------------------------------------------ in 64 bits
def axis_exponential(N, back, diag, fwd, t):
    T = torch.zeros((N, N), dtype=torch.float64, device=DEV)
    T.diagonal().fill_(t * diag)
    T.diagonal(-1).fill_(t * back)
    T.diagonal(1).fill_(t * fwd)
    return torch.linalg.matrix_exp(T)


def sine_exponential(N, t):
    """exp of t times the 1D Dirichlet Laplacian, from its sine eigenvectors."""
    k = torch.arange(1, N + 1, device=DEV, dtype=torch.float64)
    U = torch.sin(torch.outer(k, k).remainder(2 * (N + 1)) * (math.pi / (N + 1))) * math.sqrt(2.0 / (N + 1))
    lam = -4.0 * (N + 1) ** 2 * torch.sin(k * (math.pi / (2 * (N + 1)))) ** 2
    return (U * torch.exp(t * lam)) @ U


def uniformized(A, V, t):
    """exp(tA)V as a Poisson-weighted sum of powers of I + A/mu (mu the largest
    |diagonal|: no entry of the sum cancels), V of shape (n,) or (n, r)."""
    M = torch.sparse_csr_tensor(torch.from_numpy(A.row_ptr.astype(np.int64)), torch.from_numpy(A.col_idx.astype(np.int64)),
                                torch.from_numpy(A.values), (A.n, A.n)).to(DEV)
    mu = float(np.abs(A.values).max())
    z = mu * t
    X = V if V.dim() == 2 else V[:, None]
    Y = torch.zeros_like(X)
    for k in range(int(z + 12.0 * math.sqrt(z) + 40)):
        Y += math.exp(-z + k * math.log(z) - math.lgamma(k + 1)) * X
        X = X + (M @ X) / mu
    return Y if V.dim() == 2 else Y[:, 0]


def exact(case, seed):
    if case["kind"] == "batch":
        return [uniformized(A, V.T.contiguous(), t).T.contiguous().cpu().numpy() for A, V, t in batch_problems(case, seed)]
    gen = generator(seed)
    N, t = case["size"], case["t"]
    if case["matrix"] == "heat":
        v = start_vector(case, N * N, gen).view(N, N)
        E = sine_exponential(N, t)
        y = (E @ v @ E).reshape(-1)
    elif case["matrix"] == "convdiff":
        y = start_vector(case, N ** 3, gen).view(N, N, N)  # (axis 2, axis 1, axis 0)
        for d in range(3):
            E = axis_exponential(N, *convdiff_axis(N, case["pe"], d), t)
            y = torch.movedim(torch.tensordot(E, y, dims=([1], [2 - d])), 0, 2 - d)
        y = y.reshape(-1)
    else:
        A = make_matrix(case, gen)
        y = uniformized(A, start_vector(case, A.n, gen), t)
    if case["host"]:
        y = y.cpu().numpy()
    return y if case["precision"] == "mixed" else {"y": y, "accepted": None, "attempts": None}
