"""Performance cases of the library: the calls that programs make, over the sizes they make them at.

Each case is one user-level operation on a symmetric positive definite
block-tridiagonal-with-arrowhead matrix of ``n`` diagonal blocks of size
``b`` and arrow width ``a``:

* ``factor``   -- ``pobtaf`` on a fresh copy of the stacks;
* ``selinv``   -- ``pobtasi`` on a fresh copy of a factor;
* ``solve``    -- ``pobtas`` forward then backward, in place on a copy of B;
* ``refine``   -- ``pobtas_refine`` (solve and iterative refinement);
* ``workflow`` -- factor, forward and backward solve, selected inverse;
* ``grad``     -- ``bta_logdet_quad`` forward and backward;
* ``batch``    -- one replay of a ``BatchPlan`` over uneven matrices.

The library computes in place, so a pass starts by copying the inputs into
the buffers it works on.  Matrices follow the library's synthetic workloads
(uniform entries, diagonal-dominance shift); factors are drawn with the
scale the factor of such a matrix has.
"""

from __future__ import annotations

import math

import torch

import serinv_gb300 as sg
from serinv_gb300.autograd import bta_logdet_quad
from serinv_gb300.batched import BatchPlan
from serinv_gb300.refine import pobtas_refine

DEV = "cuda"
DTYPES = {"float64": torch.float64, "float32": torch.float32, "complex128": torch.complex128}


def listed():
    def case(name, op, n, b, a, nrhs=0, dtype="float64", precision="fp64", **more):
        return dict(name=name, op=op, n=n, b=b, a=a, nrhs=nrhs, dtype=dtype, precision=precision, **more)

    return [
        # the size of a unit test or a first try at the prompt: launches and latency
        case("workflow-tiny", "workflow", 4, 3, 2, 2),
        # a small model on the default precision: 128 blocks of 64, one right-hand side
        case("workflow-small", "workflow", 128, 64, 16, 1),
        # ragged sizes in single precision, a few right-hand sides
        case("workflow-f32-odd", "workflow", 75, 130, 17, 4, dtype="float32"),
        # Hermitian matrices (Green's-function style use)
        case("workflow-c128", "workflow", 24, 90, 12, 2, dtype="complex128"),
        # large blocks on the default precision, each direction by itself
        case("factor-fp64", "factor", 128, 512, 64),
        case("selinv-fp64", "selinv", 128, 512, 64),
        # the largest matrix of the benchmark in mixed precision, each direction by itself
        case("factor-mixed", "factor", 512, 512, 64, precision="mixed"),
        case("selinv-mixed", "selinv", 512, 512, 64, precision="mixed"),
        # many right-hand sides against the benchmark's factor
        case("solve-16rhs", "solve", 512, 512, 64, 16),
        # refined solve at ragged sizes
        case("refine-odd", "refine", 150, 200, 33, 3, iters=1),
        # one likelihood evaluation with its gradient
        case("grad-fp64", "grad", 128, 256, 32, 1),
        # uneven matrices side by side in one graph replay, half of them float32
        case("batch-uneven", "batch", 96, 256, 16, 4, precision="mixed", count=12),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    op = rng.choice(["factor", "selinv", "solve", "refine", "workflow", "workflow", "grad", "batch"])
    if op == "batch":
        return dict(op=op, n=rng.randint(16, 96), b=rng.choice([64, 128, 256]), a=rng.choice([0, 4, 16]),
                    nrhs=rng.randint(1, 5), dtype="float64", precision=rng.choice(["fp64", "mixed"]),
                    count=rng.randint(4, 12))
    dtype = "float64"
    if op in ("factor", "selinv", "solve", "workflow"):
        dtype = rng.choice(["float64", "float64", "float64", "float32", "complex128"])
    b = log_int(2, 256 if dtype == "complex128" else 512)
    n = log_int(3, 400)
    if op in ("workflow", "grad", "refine"):
        n = max(3, min(n, int(12e9 / b ** 3), int(8e4 / b)))
    else:
        n = max(3, min(n, int(25e9 / b ** 3)))
    if dtype == "complex128":
        n = max(3, n // 8)
    precision = rng.choice(["fp64", "mixed", "mixed:7:7"]) if dtype == "float64" and op != "solve" else "fp64"
    c = dict(op=op, n=n, b=b, a=rng.choice([0, 1]) * log_int(1, 64), nrhs=0, dtype=dtype, precision=precision)
    if op in ("solve", "refine", "workflow", "grad"):
        c["nrhs"] = log_int(1, 24)
    if op == "refine":
        c["iters"] = rng.randint(0, 2)
        c["precision"] = "fp64"
    return c


# ---- inputs -------------------------------------------------------------


def _uniform(g, dtype):
    """Uniform [-1, 1) entries (both parts of a complex type)."""
    def u(*shape):
        real = torch.float64 if dtype in (torch.float64, torch.complex128) else torch.float32
        r = torch.rand(shape, generator=g, device=DEV, dtype=real) * 2 - 1
        return torch.complex(r, torch.rand(shape, generator=g, device=DEV, dtype=real) * 2 - 1) if dtype.is_complex else r
    return u


def _matrix(c, seed):
    """Lower stacks of a diagonally dominant Hermitian matrix, and a right-hand side."""
    n, b, a, dt = c["n"], c["b"], c["a"], DTYPES[c["dtype"]]
    u = _uniform(torch.Generator(device=DEV).manual_seed(seed), dt)
    D = u(n, b, b)
    D = D + D.mH
    Lo, Ar, T = u(n - 1, b, b), u(n, a, b), u(a, a)
    T = T + T.mH
    rows = D.abs().sum(2) - torch.diagonal(D, dim1=1, dim2=2).abs()
    if n > 1:
        rows[1:] += Lo.abs().sum(2)
        rows[:-1] += Lo.abs().sum(1)
    rows += Ar.abs().sum(1)
    torch.diagonal(D, dim1=1, dim2=2).add_(1 + rows)
    torch.diagonal(T).add_(1 + T.abs().sum(1) + Ar.abs().sum((0, 2)))
    return [D, Lo, Ar, T], u(n * b + a, max(1, c["nrhs"]))


def _factor(c, seed):
    """Lower stacks of a factor with the scale of a dominant matrix's: a
    diagonal near the root of the row sums, the other entries that much
    below 1."""
    n, b, a, dt = c["n"], c["b"], c["a"], DTYPES[c["dtype"]]
    u = _uniform(torch.Generator(device=DEV).manual_seed(seed), dt)
    s = math.sqrt(1 + 1.5 * b + 0.5 * a)
    st = math.sqrt(1 + 0.5 * n * b)
    D = torch.tril(u(n, b, b), -1) / s
    torch.diagonal(D, dim1=1, dim2=2).copy_(s * (1 + 0.05 * u(n, b).real))
    Lo, Ar = u(n - 1, b, b) / s, u(n, a, b) / s
    T = torch.tril(u(a, a), -1) / st
    torch.diagonal(T).copy_(st * (1 + 0.05 * u(a).real))
    return [D, Lo, Ar, T], u(n * b + a, max(1, c["nrhs"]))


def _product(L):
    """Lower stacks of L L^H."""
    D, Lo, Ar, T = L
    A = [D @ D.mH, Lo @ D[:-1].mH, Ar @ D.mH, T @ T.mH + (Ar @ Ar.mH).sum(0)]
    A[0][1:] += Lo @ Lo.mH
    A[2][1:] += Ar[:-1] @ Lo.mH
    return A


def _items(c, seed):
    """The batch's matrices: sizes spread below (n, b) in a fixed pattern,
    every second one float32."""
    out = []
    for k in range(c["count"]):
        n = max(8, c["n"] * (c["count"] - k) // c["count"])
        b = max(32, c["b"] >> (k % 4))
        a = (c["a"], 0, 4)[k % 3]
        out.append(dict(c, n=n, b=b, a=a, dtype="float64" if k % 2 == 0 else "float32"))
    return [(i, *_matrix(i, seed * 1000 + k)) for k, i in enumerate(out)]


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["op"] == "batch":
        items = _items(c, seed)
        s["src"] = [t for _, m, B in items for t in (*m, B)]
        s["dst"] = [t.clone() for t in s["src"]]
        mats = [tuple(s["dst"][5 * k:5 * k + 4]) for k in range(len(items))]
        s["plan"] = BatchPlan(mats, [s["dst"][5 * k + 4] for k in range(len(items))],
                              precisions=[c["precision"]] * len(items), nstreams=12)
        return s
    if c["op"] in ("selinv", "solve", "refine"):
        s["src"], s["B"] = _factor(c, seed)
        if c["op"] == "refine":
            s["A"] = _product(s["src"])
    else:
        s["src"], s["B"] = _matrix(c, seed)
    if c["op"] in ("factor", "selinv", "workflow"):
        s["dst"] = [t.clone() for t in s["src"]]
    if c["op"] == "workflow":
        s["L"] = [t.clone() for t in s["src"]]
    if c["op"] == "grad":
        s["par"] = [t.requires_grad_(True) for t in (*s["src"], s["B"][:, 0].contiguous() if c["nrhs"] == 1 else s["B"])]
    s["x"] = s["B"].detach().clone()
    return s


def run(state):
    s, c = state, state["case"]
    op, prec = c["op"], c["precision"]
    if op == "batch":
        for d, x in zip(s["dst"], s["src"]):
            d.copy_(x)
        s["plan"].run()
        return s["dst"]
    if op == "grad":
        loss = bta_logdet_quad(*s["par"], precision=prec)
        return [loss.detach(), *torch.autograd.grad(loss, s["par"])]
    if op == "solve":
        s["x"].copy_(s["B"])
        sg.pobtas(*s["src"], s["x"], trans="N")
        sg.pobtas(*s["src"], s["x"], trans="C")
        return s["x"]
    if op == "refine":
        s["x"].copy_(s["B"])
        pobtas_refine(*s["A"], *s["src"], s["x"], iters=c["iters"])
        return s["x"]
    for d, x in zip(s["dst"], s["src"]):
        d.copy_(x)
    if op == "factor":
        sg.pobtaf(*s["dst"], precision=prec)
        return s["dst"]
    if op == "selinv":
        sg.pobtasi(*s["dst"], precision=prec)
        return s["dst"]
    sg.pobtaf(*s["dst"], precision=prec)  # workflow
    for d, x in zip(s["L"], s["dst"]):
        d.copy_(x)
    s["x"].copy_(s["B"])
    sg.pobtas(*s["dst"], s["x"], trans="N", precision=prec)
    sg.pobtas(*s["dst"], s["x"], trans="C", precision=prec)
    sg.pobtasi(*s["dst"], precision=prec)
    return [s["L"], s["x"], s["dst"]]


# ---- the work a pass cannot do without ---------------------------------------


def work(case):
    c = case
    if c["op"] == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for k in range(c["count"]):
            w = work(dict(c, op="workflow", n=max(8, c["n"] * (c["count"] - k) // c["count"]), b=max(32, c["b"] >> (k % 4)),
                          a=(c["a"], 0, 4)[k % 3], dtype="float64" if k % 2 == 0 else "float32"))
            tot = {q: tot[q] + w[q] for q in tot}
        return tot
    n, b, a, r, op = c["n"], c["b"], c["a"], c["nrhs"], c["op"]
    item = {"float64": 8, "float32": 4, "complex128": 16}[c["dtype"]]
    mul = 4 if c["dtype"] == "complex128" else 1
    mat = item * (n * b * b + (n - 1) * b * b + n * a * b + a * a)
    vec = item * (n * b + a) * r
    fac = n * (7 / 3 * b ** 3 + 3 * a * b * b + a * a * b) + a ** 3 / 3
    inv = n * (19 / 3 * b ** 3 + 7 * a * b * b + 2 * a * a * b) + 4 * a ** 3 / 3
    sol = 2 * r * (n * b * b + 2 * (n - 1) * b * b + 2 * n * a * b + a * a)
    if op == "factor":
        return {"bytes": 2 * mat, "flops": mul * fac}
    if op == "selinv":
        return {"bytes": 2 * mat, "flops": mul * inv}
    if op == "solve":
        return {"bytes": mat + 2 * vec, "flops": mul * sol}
    if op == "refine":
        return {"bytes": 2 * mat + 2 * vec, "flops": mul * sol * (1 + 2 * c["iters"])}
    if op == "grad":
        return {"bytes": 2 * mat + 2 * vec, "flops": mul * (fac + inv + sol)}
    return {"bytes": 3 * mat + 2 * vec, "flops": mul * (fac + inv + sol)}


# ---- the same values in 64 bits, by plain torch --------------------------------


def _wide(ts):
    return [t.detach().to(torch.complex128 if t.is_complex() else torch.float64) for t in ts]


def _trs(L, B):
    """L^{-1} B."""
    return torch.linalg.solve_triangular(L, B, upper=False)


def _pobtaf(D, Lo, Ar, T):
    D, Lo, Ar, T = (t.clone() for t in (D, Lo, Ar, T))
    n, a = D.shape[0], T.shape[0]
    for i in range(n):
        D[i] = torch.linalg.cholesky(D[i])
        if i < n - 1:
            Lo[i] = _trs(D[i], Lo[i].mH.contiguous()).mH
            D[i + 1] -= Lo[i] @ Lo[i].mH
        if a:
            Ar[i] = _trs(D[i], Ar[i].mH.contiguous()).mH
            T -= Ar[i] @ Ar[i].mH
            if i < n - 1:
                Ar[i + 1] -= Ar[i] @ Lo[i].mH
    if a:
        T = torch.linalg.cholesky(T)
    return [D, Lo, Ar, T]


def _pobtasi(D, Lo, Ar, T):
    D, Lo, Ar, T = (t.clone() for t in (D, Lo, Ar, T))
    n, b, a = D.shape[0], D.shape[1], T.shape[0]
    eye = torch.eye(b, dtype=D.dtype, device=D.device)
    if a:
        Ti = _trs(T, torch.eye(a, dtype=D.dtype, device=D.device))
        T = Ti.mH @ Ti
    for i in range(n - 1, -1, -1):
        Li = _trs(D[i], eye)
        X = Li.mH.clone()
        lo = Lo[i].clone() if i < n - 1 else None
        ar = Ar[i].clone()
        if lo is not None:
            Lo[i] = -(D[i + 1] @ lo + Ar[i + 1].mH @ ar) @ Li
            Ar[i] = -(Ar[i + 1] @ lo + T @ ar) @ Li
            X -= Lo[i].mH @ lo
        else:
            Ar[i] = -(T @ ar) @ Li
        X -= Ar[i].mH @ ar
        D[i] = X @ Li
    return [D, Lo, Ar, T]


def _pobtas(D, Lo, Ar, T, B, steps="NC"):
    n, b, a = D.shape[0], D.shape[1], T.shape[0]
    x = B.reshape(B.shape[0], -1).clone()
    if "N" in steps:
        for i in range(n):
            k = slice(i * b, (i + 1) * b)
            x[k] = _trs(D[i], x[k].contiguous())
            if i < n - 1:
                x[k.stop:k.stop + b] -= Lo[i] @ x[k]
            x[n * b:] -= Ar[i] @ x[k]
        if a:
            x[n * b:] = _trs(T, x[n * b:].contiguous())
    if "C" in steps:
        if a:
            x[n * b:] = torch.linalg.solve_triangular(T.mH, x[n * b:].contiguous(), upper=True)
        for i in range(n - 1, -1, -1):
            k = slice(i * b, (i + 1) * b)
            r = x[k] - Ar[i].mH @ x[n * b:]
            if i < n - 1:
                r = r - Lo[i].mH @ x[k.stop:k.stop + b]
            x[k] = torch.linalg.solve_triangular(D[i].mH, r.contiguous(), upper=True)
    return x.reshape(B.shape)


def _pattern(X, x, dtype):
    """d(logdet + quadratic form)/d(stacks) from the selected inverse X and the solution x."""
    D, Lo, Ar, T = X
    n, b = D.shape[0], D.shape[1]
    xb, xt = x[:n * b].reshape(n, b, -1), x[n * b:]
    G = [D - xb @ xb.mT, Lo - xb[1:] @ xb[:-1].mT, Ar - xt @ xb.mT, T - xt @ xt.mT]
    G[0] = torch.tril(G[0], -1) * 2 + torch.diag_embed(torch.diagonal(G[0], dim1=1, dim2=2))
    G[3] = torch.tril(G[3], -1) * 2 + torch.diag(torch.diagonal(G[3]))
    return [G[0], G[1] * 2, G[2] * 2, G[3]]


def exact(case, seed):
    c = case
    if c["op"] == "batch":
        out = []
        for _, m, B in _items(c, seed):
            L = _pobtaf(*_wide(m))
            out += [*_pobtasi(*L), _pobtas(*L, *_wide([B]))]
        return out
    if c["op"] in ("selinv", "solve", "refine"):
        L, B = _factor(c, seed)
        if c["op"] == "selinv":
            return _pobtasi(*_wide(L))
        if c["op"] == "solve":
            return _pobtas(*_wide(L), *_wide([B]))
        L = _pobtaf(*_product(_wide(L)))
        return _pobtas(*L, *_wide([B]))
    m, B = _matrix(c, seed)
    m = _wide(m)
    L = _pobtaf(*m)
    if c["op"] == "factor":
        return L
    B = _wide([B])[0]
    if c["op"] == "workflow":
        return [L, _pobtas(*L, B), _pobtasi(*L)]
    y = B[:, 0] if c["nrhs"] == 1 else B
    x = _pobtas(*L, y)
    loss = 2 * torch.log(torch.diagonal(L[0], dim1=1, dim2=2)).sum() + (y * x).sum()
    if c["a"]:
        loss = loss + 2 * torch.log(torch.diagonal(L[3])).sum()
    return [loss, *_pattern(_pobtasi(*L), x.reshape(x.shape[0], -1), y.dtype), 2 * x]
