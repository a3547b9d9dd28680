"""Performance cases: the work a program has this library do, through its
public entry points, over the range of sizes it meets.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a program holds before the call: operands on the
                       device (host arrays for the host entry), a grouped plan
  run(state)           one pass; its outputs
  work(case)           bytes and FLOPs the pass cannot do without
  exact(case, seed)    the outputs as plain torch gives them in 64 bits

Kinds of case:
  gemm      C = alpha op(A) op(B) + beta C on device operands (Context.dgemm_device),
            native FP64 or the library's own choice of route (AUTO)
  adjoint   the reverse of a GEMM (Context.adjoint_device)
  grouped   a batch of uneven GEMMs through a captured plan (Context.grouped_plan)
  qr        blocked Householder QR and its thin Q (qr_factor_device, qr_build_q_device)
  hess      Hessenberg reduction with Q (hessenberg_device)
  bidiag    Golub-Kahan bidiagonalisation with U and V (bidiag_device)
  host      OptimizedBLAS3.gemm on host matrices, copies included

The factorisations work in place, so a pass first copies the caller's matrix
into the work array, as a program that keeps its matrix does.
"""
import math

import numpy as np
import torch

import jlc_b200 as jlc

PRECISION = {"native": jlc.JLC_PREC_NATIVE, "auto": jlc.JLC_PREC_AUTO}
LAYOUT = {"row": jlc.JLC_ROW_MAJOR, "col": jlc.JLC_COL_MAJOR}


def _gemm(name, m, n, k, la="row", lb="row", pad=0, alpha=1.0, beta=0.0, precision="native"):
    c = {"kind": "gemm", "m": m, "n": n, "k": k, "la": la, "lb": lb, "pad": pad, "alpha": alpha, "beta": beta,
         "precision": precision}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one small product per call, the SMALL dispatch class: launches and host latency count
        _gemm("gemm small", 96, 80, 112),
        # a plain dense product with alpha and beta, the reference's benchmark size
        _gemm("gemm 1024", 1024, 1024, 1024, alpha=1.5, beta=0.5),
        # A^T B on odd sizes with odd leading dimensions: sub-blocks of larger matrices
        _gemm("gemm ragged transa", 1999, 1501, 2743, la="col", pad=2),
        # a medium product on the automatic route, column-major B
        _gemm("gemm auto 3000", 3000, 2304, 2600, lb="col", precision="auto"),
        # the headline product on the automatic route
        _gemm("gemm auto 8192", 8192, 8192, 8192, precision="auto"),
        # matrix times vector
        _gemm("matvec 16384", 16384, 1, 16384),
        # the backward pass of C = A B + C
        {"name": "adjoint", "kind": "adjoint", "m": 4096, "n": 4096, "k": 2048, "alpha": 1.0, "beta": 1.0,
         "precision": "native"},
        # 20,000 uneven products in one captured launch
        {"name": "grouped 20000", "kind": "grouped", "count": 20000},
        # least squares: QR of a tall matrix and its thin Q
        {"name": "qr 2304x2048", "kind": "qr", "m": 2304, "n": 2048},
        # the first stage of a dense eigenvalue computation
        {"name": "hessenberg 1024", "kind": "hess", "n": 1024},
        # the first stage of a dense SVD
        {"name": "bidiag 1152x1024", "kind": "bidiag", "m": 1152, "n": 1024},
        # the drop-in host entry on heap matrices, copies both ways
        {"name": "host gemm", "kind": "host", "m": 1536, "n": 1280, "k": 1400, "alpha": 1.0, "beta": 0.0},
    ]


def _size(rng, lo, hi):
    """A size, even in its logarithm; every third one on a multiple of 64 where there is room."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 1 / 3 and v >= 128:
        v = v // 64 * 64
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "auto", "matvec", "adjoint", "grouped", "qr", "hess", "bidiag", "host"])
    if kind == "gemm":
        return _gemm(None, _size(rng, 24, 4096), _size(rng, 24, 4096), _size(rng, 24, 4096), rng.choice(["row", "col"]),
                     rng.choice(["row", "col"]), rng.choice([0, 0, 1, 6]), rng.choice([1.0, -1.0, 1.5]),
                     rng.choice([0.0, 0.5, 1.0]))
    if kind == "auto":
        return _gemm(None, _size(rng, 2048, 6144), _size(rng, 2048, 6144), _size(rng, 1024, 8192),
                     rng.choice(["row", "col"]), rng.choice(["row", "col"]), rng.choice([0, 0, 1, 6]),
                     rng.choice([1.0, -1.0]), rng.choice([0.0, 0.5]), "auto")
    if kind == "matvec":
        m, k = _size(rng, 512, 16384), _size(rng, 512, 16384)
        return _gemm(None, m, 1, k, rng.choice(["row", "col"])) if rng.random() < 0.75 else \
            _gemm(None, 1, m, k, "row", rng.choice(["row", "col"]))
    if kind == "adjoint":
        return {"kind": "adjoint", "m": _size(rng, 256, 4096), "n": _size(rng, 256, 4096), "k": _size(rng, 256, 2048),
                "alpha": rng.choice([1.0, 1.5]), "beta": rng.choice([1.0, 0.5]),
                "precision": rng.choice(["native", "auto"])}
    if kind == "grouped":
        return {"kind": "grouped", "count": _size(rng, 500, 19999)}
    if kind == "qr":
        n = _size(rng, 64, 2048)
        return {"kind": "qr", "m": min(2304, n + int(n * rng.choice([0, 0.125, 0.5]))), "n": n}
    if kind == "hess":
        return {"kind": "hess", "n": _size(rng, 64, 1023)}
    if kind == "bidiag":
        n = _size(rng, 64, 1023)
        return {"kind": "bidiag", "m": min(1152, n + int(n * rng.choice([0, 0.125, 0.5]))), "n": n}
    return {"kind": "host", "m": _size(rng, 64, 1535), "n": _size(rng, 64, 1535), "k": _size(rng, 64, 1535),
            "alpha": rng.choice([1.0, -1.0]), "beta": rng.choice([0.0, 0.5])}


# ---------------------------------------------------------------- operands
_STREAM = []


def _context():
    """The thread's context on a stream of the program's own, which torch's copies share."""
    ctx = jlc.default_context()
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    ctx.set_stream(_STREAM[0].cuda_stream)
    return ctx, _STREAM[0]


class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, *shape):
        """FP64 on [-1, 1)."""
        return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=self.g) * 2 - 1

    def normal(self, *shape):
        return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=self.g)


def _gemm_operands(case, seed):
    """op(A) stored rows x (cols + pad), op(B) likewise, C dense."""
    r = _Random(seed)
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    a = r.uniform(*((m, k + pad) if case["la"] == "row" else (k, m + pad)))
    b = r.uniform(*((k, n + pad) if case["lb"] == "row" else (n, k + pad)))
    c = r.uniform(m, n) if case["beta"] else torch.zeros(m, n, dtype=torch.float64, device="cuda")
    return a, b, c


def _adjoint_operands(case, seed):
    r = _Random(seed)
    m, n, k = case["m"], case["n"], case["k"]
    return r.normal(m, k), r.normal(k, n), r.normal(m, n), r.normal(m, n)


def _grouped_problems(case, seed):
    """30 % tiny (M = N = K in {2, 3, 4}), 70 % with M, N, K log-uniform on
    [8, 512]; alpha on [-2, 2], beta on [-1, 1] so that repeated updates stay
    finite.  The shapes are the batch's, the entries the seed's."""
    g = np.random.default_rng(case["count"])
    problems, off = [], 0
    for _ in range(case["count"]):
        if g.random() < 0.3:
            m = n = k = int(g.integers(2, 5))
        else:
            m, n, k = (int(x) for x in np.exp(g.uniform(np.log(8), np.log(512), size=3)).round())
        even = [(x + 1) // 2 * 2 for x in (m * k, k * n, m * n)]
        problems.append((m, n, k, float(g.uniform(-2, 2)), float(g.uniform(-1, 1)), off, off + even[0]))
        off += even[0] + even[1]
    coff, cs = 0, []
    for m, n, *_ in problems:
        cs.append(coff)
        coff += (m * n + 1) // 2 * 2
    r = _Random(seed)
    return problems, cs, r.uniform(off), r.uniform(coff)


def _square(case, seed):
    """The column-major input: row j of the array is column j of the matrix."""
    return _Random(seed).uniform(case["n"], case.get("m", case["n"]))


def _host_operands(case, seed):
    g = np.random.default_rng(int(seed))
    m, n, k = case["m"], case["n"], case["k"]
    return tuple(g.uniform(-1.0, 1.0, s) for s in (m * k, k * n, m * n))


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "host":
        a, b, c = _host_operands(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        s.update(a=jlc.Matrix.wrap(a, m, k), b=jlc.Matrix.wrap(b, k, n), c=jlc.Matrix.wrap(c, m, n))
        return s
    s["ctx"], s["stream"] = _context()
    if kind == "gemm":
        s["a"], s["b"], s["c"] = _gemm_operands(case, seed)
    elif kind == "adjoint":
        s["a"], s["b"], s["c"], s["dc"] = _adjoint_operands(case, seed)
        s["out"] = [torch.empty_like(s["a"]), torch.empty_like(s["b"]), torch.empty(1, dtype=torch.float64, device="cuda"),
                    torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty_like(s["c"])]
    elif kind == "grouped":
        problems, cs, s["ab"], s["c"] = _grouped_problems(case, seed)
        torch.cuda.current_stream().synchronize()
        ab, c = s["ab"].data_ptr(), s["c"].data_ptr()
        s["plan"] = s["ctx"].grouped_plan(
            [dict(m=m, n=n, k=k, layout_a=0, layout_b=0, lda=k, ldb=n, ldc=n, alpha=alpha, beta=beta, a=ab + 8 * pa,
                  b=ab + 8 * pb, c=c + 8 * pc) for (m, n, k, alpha, beta, pa, pb), pc in zip(problems, cs)], graph=True)
    else:
        s["a0"] = _square(case, seed)
        n, m = s["a0"].shape
        new = lambda *shape: torch.empty(*shape, dtype=torch.float64, device="cuda")  # noqa: E731
        s["a"] = torch.empty_like(s["a0"])
        if kind == "qr":
            s["tau"], s["q"] = new(n), new(n, m)
        elif kind == "hess":
            s["q"] = new(n, n)
        else:
            s["d"], s["e"], s["u"], s["v"] = new(n), new(n - 1), new(m, m), new(n, n)
    torch.cuda.current_stream().synchronize()
    return s


# ---------------------------------------------------------------- run
def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "host":
        jlc.OptimizedBLAS3.gemm(s["a"], s["b"], s["c"], case["alpha"], case["beta"])
        return s["c"].getRawData()
    ctx = s["ctx"]
    if kind == "gemm":
        ctx.dgemm_device(LAYOUT[case["la"]], LAYOUT[case["lb"]], case["m"], case["n"], case["k"], case["alpha"],
                         s["a"].data_ptr(), s["a"].shape[1], s["b"].data_ptr(), s["b"].shape[1], case["beta"],
                         s["c"].data_ptr(), case["n"], PRECISION[case["precision"]], report=False)
        return s["c"]
    if kind == "adjoint":
        m, n, k = case["m"], case["n"], case["k"]
        da, db, dalpha, dbeta, dc_in = s["out"]
        ctx.adjoint_device(m, n, k, case["alpha"], case["beta"], s["a"].data_ptr(), k, s["b"].data_ptr(), n,
                           s["c"].data_ptr(), n, s["dc"].data_ptr(), n, da.data_ptr(), k, db.data_ptr(), n,
                           dalpha.data_ptr(), dbeta.data_ptr(), dc_in.data_ptr(), n, PRECISION[case["precision"]])
        return {"da": da, "db": db, "dalpha": dalpha, "dbeta": dbeta, "dc_in": dc_in}
    if kind == "grouped":
        s["plan"].run()
        return s["c"]
    a = s["a"]
    n, m = a.shape
    with torch.cuda.stream(s["stream"]):
        a.copy_(s["a0"])
    if kind == "qr":
        ctx.qr_factor_device(m, n, a.data_ptr(), m, s["tau"].data_ptr())
        ctx.qr_build_q_device(m, n, n, a.data_ptr(), m, s["tau"].data_ptr(), s["q"].data_ptr(), m)
        return {"f": a, "tau": s["tau"], "q": s["q"]}
    if kind == "hess":
        ctx.hessenberg_device(n, a.data_ptr(), n, s["q"].data_ptr(), n)
        return {"h": a, "q": s["q"]}
    ctx.bidiag_device(m, n, a.data_ptr(), m, s["d"].data_ptr(), s["e"].data_ptr(), s["u"].data_ptr(), m,
                      s["v"].data_ptr(), n)
    return {"d": s["d"], "e": s["e"], "u": s["u"], "v": s["v"], "f": a}


# ---------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    m, n, k = case.get("m", 0), case.get("n", 0), case.get("k", 0)
    if kind in ("gemm", "host"):
        return {"bytes": 8.0 * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2.0 * m * n * k}
    if kind == "adjoint":  # A, B, C, dC read once; dA, dB, dC_in written once; two products and two dots
        return {"bytes": 8.0 * (2 * m * k + 2 * k * n + 3 * m * n), "flops": 4.0 * m * n * k + 2.0 * (m * k + m * n)}
    if kind == "grouped":
        g = np.random.default_rng(case["count"])
        total, flops = 0.0, 0.0
        for _ in range(case["count"]):  # the same draws as _grouped_problems
            if g.random() < 0.3:
                m = n = k = int(g.integers(2, 5))
            else:
                m, n, k = (int(x) for x in np.exp(g.uniform(np.log(8), np.log(512), size=3)).round())
            g.uniform(), g.uniform()
            total += 8.0 * (m * k + k * n + 2 * m * n)
            flops += 2.0 * m * n * k
        return {"bytes": total, "flops": flops}
    if kind == "qr":  # the factorisation and the thin Q
        return {"bytes": 8.0 * 3 * m * n, "flops": 2.0 * (2.0 * m * n * n - 2.0 / 3.0 * n ** 3)}
    if kind == "hess":
        return {"bytes": 8.0 * 3 * n * n, "flops": 14.0 / 3.0 * n ** 3}
    # B, U (m x m) and V
    return {"bytes": 8.0 * (2 * m * n + m * m + n * n),
            "flops": 4.0 * n * n * (m - n / 3.0) + 4.0 * (m * m * n - m * n * n + n ** 3 / 3.0) + 4.0 / 3.0 * n ** 3}


# ---------------------------------------------------------------- exact
def _reflect(x):
    """v (v_0 = 1), tau and beta of the Householder reflector that takes x to beta e_0."""
    norm = torch.linalg.vector_norm(x)
    beta = torch.where(x[0] >= 0, -norm, norm)
    v = x / (x[0] - beta)
    v[0] = 1.0
    return v, (beta - x[0]) / beta, beta


def _hessenberg(h):
    n = h.shape[0]
    q = torch.eye(n, dtype=h.dtype, device=h.device)
    for k in range(n - 2):
        v, tau, _ = _reflect(h[k + 1:, k].clone())
        h[k + 1:, k:] -= torch.outer(v * tau, v @ h[k + 1:, k:])
        h[:, k + 1:] -= torch.outer(h[:, k + 1:] @ v, v * tau)
        q[:, k + 1:] -= torch.outer(q[:, k + 1:] @ v, v * tau)
    return torch.triu(h, -1), q


def _bidiagonal(a):
    """d, e, U, V and the factored matrix, whose diagonal and superdiagonal keep the reflected vectors' first entries."""
    m, n = a.shape
    new = lambda k: torch.eye(k, dtype=a.dtype, device=a.device)  # noqa: E731
    u, v = new(m), new(n)
    d, e = torch.empty(n, dtype=a.dtype, device=a.device), torch.empty(n - 1, dtype=a.dtype, device=a.device)
    for k in range(n):
        x, tau, d[k] = _reflect(a[k:, k].clone())
        a[k:, k + 1:] -= torch.outer(x, tau * (x @ a[k:, k + 1:]))
        u[:, k:] -= torch.outer(u[:, k:] @ x, tau * x)
        a[k + 1:, k] = x[1:]
        if k + 1 < n:
            x, tau, e[k] = _reflect(a[k, k + 1:].clone())
            a[k + 1:, k + 1:] -= torch.outer(tau * (a[k + 1:, k + 1:] @ x), x)
            v[:, k + 1:] -= torch.outer(v[:, k + 1:] @ x, tau * x)
            a[k, k + 2:] = x[1:]
    return d, e, u, v, a


def exact(case, seed):
    kind = case["kind"]
    m, n, k = case.get("m", 0), case.get("n", 0), case.get("k", 0)
    if kind == "gemm":
        a, b, c = _gemm_operands(case, seed)
        a = a[:, :k] if case["la"] == "row" else a[:, :m].T
        b = b[:, :n] if case["lb"] == "row" else b[:, :k].T
        return case["alpha"] * (a @ b) + case["beta"] * c
    if kind == "host":
        a, b, c = (torch.from_numpy(x).cuda().reshape(s) for x, s in
                   zip(_host_operands(case, seed), ((m, k), (k, n), (m, n))))
        return (case["alpha"] * (a @ b) + case["beta"] * c).reshape(-1).cpu().numpy()
    if kind == "adjoint":
        a, b, c, dc = _adjoint_operands(case, seed)
        g = dc @ b.T
        return {"da": case["alpha"] * g, "db": case["alpha"] * (a.T @ dc), "dalpha": (a * g).sum().reshape(1),
                "dbeta": (dc * c).sum().reshape(1), "dc_in": case["beta"] * dc}
    if kind == "grouped":
        problems, cs, ab, c = _grouped_problems(case, seed)
        for (m, n, k, alpha, beta, pa, pb), pc in zip(problems, cs):
            out = c[pc:pc + m * n].view(m, n)
            out.mul_(beta).add_(ab[pa:pa + m * k].view(m, k) @ ab[pb:pb + k * n].view(k, n), alpha=alpha)
        return c
    a = _square(case, seed).T
    if kind == "qr":
        f, tau = torch.geqrf(a.cpu().contiguous())
        q = torch.linalg.householder_product(f, tau)
        return {"f": f.T.contiguous(), "tau": tau, "q": q.T.contiguous()}
    if kind == "hess":
        h, q = _hessenberg(a.contiguous())
        return {"h": h.T.contiguous(), "q": q.T.contiguous()}
    d, e, u, v, f = _bidiagonal(a.contiguous())
    return {"d": d, "e": e, "u": u.T.contiguous(), "v": v.T.contiguous(), "f": f.T.contiguous()}
