"""The calls this library is timed on: what its users run, through its public
entry points, over the sizes it is meant for.

listed() names the fixed cases, draw() gives further ones from the same
ranges, prepare() makes a case's device buffers from a seed, run() is one call
as a program makes it, work() the bytes and operations of the call, and
exact() its result from plain torch in 64 bits.
"""
from __future__ import annotations

import torch

import caps_gb300 as cg

DEV = "cuda"


def listed():
    return [
        # the smallest calls: the reference's known-answer fixtures (n = 28..392,
        # integers, one 'd' or 'b' step per level), where launches are the time
        dict(name="fixture_n56_dd", op="multiply", n=56, r=2, bs=1, pattern="dd", form="plain", data="int9"),
        # a fixture with blocked leaves (-b 7): leaves repacked before and after the product
        dict(name="fixture_n392_b7", op="multiply", n=392, r=2, bs=7, pattern="bd", form="split", data="int9"),
        # one base-case product of an uneven batch's smallest class
        dict(name="leaf_m448", op="leaf", n=448, form="split", data="uniform"),
        # a mid-size multiply with leaves that fill no tile evenly
        dict(name="split_n1792", op="multiply", n=1792, r=1, bs=1, pattern="", form="split", data="uniform"),
        # leaves above 2048, which run as digit slices; ragged in every tile size
        dict(name="split_n5000", op="multiply", n=5000, r=1, bs=1, pattern="", form="split", data="uniform"),
        # the headline benchmark: n = 16384, three levels, split form
        dict(name="split_n16384", op="multiply", n=16384, r=3, bs=1, pattern="", form="split", data="uniform"),
        # integer data under a mixed pattern, as the large memory-bounded runs use it
        dict(name="split_n16384_int", op="multiply", n=16384, r=4, bs=1, pattern="bbdd", form="split", data="int1024"),
        # FP64 throughout, memory-lean steps
        dict(name="plain_n4096_dd", op="multiply", n=4096, r=2, bs=1, pattern="dd", form="plain", data="uniform"),
        # the trailing update of a Cholesky factorisation, rows spanning 40 binades
        dict(name="chol_n6144", op="chol", n=6144, r=2, alpha=1.0, form="split", data="wide"),
        # the rectangular product, two levels of blocking
        dict(name="rect_4096", op="rect", m=4096, n=3072, k=2048, div="2,1,1,1,3,1", data="uniform"),
        # column-major into the recursive layout and back, around every multiply of column-major data
        dict(name="layout_n8192", op="layout", n=8192, r=3, bs=1, data="uniform"),
        # independent multiplies of uneven sizes in one call
        dict(name="batched_uneven", op="batched", sizes="448*12,896*6,1792*3", form="split", data="uniform"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _block(rng, m):
    """A leaf block size: 1 (plain column-major leaves) or a divisor of the leaf."""
    divisors = [d for d in range(2, min(m, 64) + 1) if m % d == 0]
    return rng.choice(divisors) if divisors and rng.random() < 0.5 else 1


def _pattern(rng, r):
    return "".join(rng.choice("bd") for _ in range(r)) if rng.random() < 0.6 else ""


def draw(rng):
    kind = rng.choice(["small", "leaf", "split", "split", "split", "digits", "plain", "chol", "rect", "layout",
                       "batched"])
    if kind == "small":
        r = rng.randint(1, 3)
        m = _log_int(rng, 7, 448 >> r)
        return dict(op="multiply", n=m << r, r=r, bs=_block(rng, m), pattern=_pattern(rng, r),
                    form=rng.choice(["plain", "split"]), data=rng.choice(["int9", "uniform"]))
    if kind == "leaf":
        return dict(op="leaf", n=_log_int(rng, 32, 2048), form=rng.choice(["split", "split", "plain"]),
                    data=rng.choice(["uniform", "wide", "int1024"]))
    if kind == "split":
        r = rng.randint(1, 4)
        m = _log_int(rng, 192, min(2048, 16384 >> r))
        return dict(op="multiply", n=m << r, r=r, bs=1, pattern=_pattern(rng, r), form="split",
                    data=rng.choice(["uniform", "uniform", "wide", "int1024"]))
    if kind == "digits":
        r = rng.randint(0, 1)
        return dict(op="multiply", n=rng.randint(2049, 3000) << r, r=r, bs=1, pattern=_pattern(rng, r), form="split",
                    data=rng.choice(["uniform", "int1024"]))
    if kind == "plain":
        r = rng.randint(1, 2)
        m = _log_int(rng, 150, 1024)
        return dict(op="multiply", n=m << r, r=r, bs=1, pattern=_pattern(rng, r), form="plain",
                    data=rng.choice(["uniform", "wide", "int1024"]))
    if kind == "chol":
        r = rng.randint(0, 3)
        m = _log_int(rng, 128, min(2048, 8192 >> r))
        return dict(op="chol", n=m << r, r=r, alpha=rng.choice([1.0, 1.0, 0.0, -0.5]), form="split",
                    data=rng.choice(["uniform", "wide"]))
    if kind == "rect":
        div = rng.choice(["", "2,1,1", "1,3,1", "2,1,1,1,3,1", "4,1,1,1,2,1"])
        step = 12
        m, n, k = (step * _log_int(rng, 20, 340) for _ in range(3))
        return dict(op="rect", m=m, n=n, k=min(k, 2400), div=div, data="uniform")
    if kind == "layout":
        r = rng.randint(0, 3)
        m = _log_int(rng, 100, 8192 >> r)
        return dict(op="layout", n=m << r, r=r, bs=_block(rng, m), data="uniform")
    return dict(op="batched", sizes="448*%d,896*%d,1792*%d" % (rng.randint(1, 24), rng.randint(1, 8), rng.randint(1, 4)),
                form="split", data=rng.choice(["uniform", "int1024"]))


# ------------------------------------------------------------------ inputs
def _values(kind, count, gen):
    if kind.startswith("int"):
        lim = int(kind[3:])
        return torch.randint(-lim, lim + 1, (count,), device=DEV, generator=gen).double()
    x = torch.rand(count, dtype=torch.float64, device=DEV, generator=gen)
    x.mul_(2.0).sub_(1.0)
    if kind == "wide":  # u 2^k, k uniform in [-20, 20]
        x = torch.ldexp(x, torch.randint(-20, 21, (count,), device=DEV, generator=gen))
    return x


def _sizes(case):
    out = []
    for part in case["sizes"].split(","):
        n, count = part.split("*")
        out += [int(n)] * int(count)
    return out


def _div(case):
    return [int(x) for x in case["div"].split(",")] if case["div"] else []


def _inputs(case, seed):
    """The input values alone, in the order prepare() hands them over."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["data"]
    if case["op"] == "rect":
        return [_values(kind, a * b, gen) for a, b in ((case["m"], case["k"]), (case["k"], case["n"]))]
    if case["op"] == "layout":
        return [_values(kind, case["n"] ** 2, gen)]
    if case["op"] == "batched":
        return [(_values(kind, n * n, gen), _values(kind, n * n, gen)) for n in _sizes(case)]
    return [_values(kind, case["n"] ** 2, gen) for _ in range(3 if case["op"] == "chol" else 2)]


def prepare(case, seed):
    x = _inputs(case, seed)
    s = {"case": case, "in": x}
    op = case["op"]
    if op == "rect":
        s["C"] = torch.zeros(case["m"] * case["n"], dtype=torch.float64, device=DEV)
    elif op == "batched":
        s["As"], s["Bs"] = [a for a, _ in x], [b for _, b in x]
        s["Cs"] = [torch.empty_like(a) for a, _ in x]
        s["ns"] = _sizes(case)
    elif op == "layout":
        s["desc"] = cg.MatDescriptor.make(case["n"], case["r"], case["bs"])
        s["caps"], s["back"] = torch.empty_like(x[0]), torch.empty_like(x[0])
    else:
        s["C"] = torch.empty_like(x[0])
        if op == "multiply":
            s["desc"] = cg.MatDescriptor.make(case["n"], case["r"], case["bs"])
    return s


def run(s):
    case, x = s["case"], s["in"]
    op = case["op"]
    if op == "multiply":
        cg.multiply(x[0], x[1], s["C"], s["desc"], case["pattern"] or None, form=case["form"])
        return s["C"]
    if op == "leaf":
        cg.leaf_gemm(x[0], x[1], s["C"], case["n"], form=case["form"])
        return s["C"]
    if op == "chol":
        if case["alpha"] != 0.0:
            s["C"].copy_(x[2])  # the update is in place: each pass starts from the same trailing matrix
        cg.chol_mult(s["C"], x[0], x[1], case["n"], case["r"], case["alpha"], form=case["form"])
        return s["C"]
    if op == "rect":
        div = _div(case)
        r = len(div) // 3
        cg.rect_mm(x[0], x[1], s["C"], case["m"], case["n"], case["k"], r, "d" * r, div)
        return s["C"]
    if op == "layout":
        cg.to_caps_layout(x[0], s["caps"], s["desc"])
        cg.from_caps_layout(s["caps"], s["back"], s["desc"])
        return [s["caps"], s["back"]]
    cg.multiply_batched(s["As"], s["Bs"], s["Cs"], s["ns"], form=case["form"])
    return s["Cs"]


def work(case):
    """Each operand read once and each result written once; the multiply-adds
    of the leaf products the recursion cannot do without (7^r of them)."""
    op = case["op"]
    if op == "layout":
        return {"bytes": 32 * case["n"] ** 2, "flops": 0}
    if op == "rect":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if op == "batched":
        return {"bytes": sum(24 * n * n for n in _sizes(case)), "flops": sum(2 * n ** 3 for n in _sizes(case))}
    n, r = case["n"], case.get("r", 0)
    arrays = 4 if op == "chol" and case["alpha"] != 0.0 else 3
    return {"bytes": 8 * arrays * n * n, "flops": 7 ** r * 2 * (n >> r) ** 3}


# ------------------------------------------------------------------ 64-bit results
def _unpack(x, n, r, bs):
    """The recursive block layout as an n x n matrix: quadrants 11, 21, 12, 22
    per level, then column-major blocks, column-major inside."""
    m = n >> r
    b = m if bs == 1 else bs
    k = r + 2
    dims = [2, 2] * r + [m // b, m // b, b, b]  # (column, row) pairs, outermost first
    return x.reshape(dims).permute([2 * i + 1 for i in range(k)] + [2 * i for i in range(k)]).reshape(n, n)


def _pack(X, n, r, bs):
    m = n >> r
    b = m if bs == 1 else bs
    k = r + 2
    dims = [2] * r + [m // b, b]
    return X.reshape(dims + dims).permute([j for i in range(k) for j in (k + i, i)]).reshape(-1)


def _rect_unpack(x, rows, cols, grid):
    """Nested column-major grids of blocks, the innermost blocks column-major."""
    if not grid:
        return x.reshape(cols, rows).t()
    (dr, dc), h, w = grid[0], rows // grid[0][0], cols // grid[0][1]
    parts = x.reshape(dc, dr, h * w)
    return torch.cat([torch.cat([_rect_unpack(parts[j, i], h, w, grid[1:]) for i in range(dr)], 0)
                      for j in range(dc)], 1)


def _rect_pack(X, grid):
    if not grid:
        return X.t().reshape(-1)
    dr, dc = grid[0]
    return torch.cat([_rect_pack(b, grid[1:]) for col in X.chunk(dc, 1) for b in col.chunk(dr, 0)])


def exact(case, seed):
    x = _inputs(case, seed)
    op = case["op"]
    if op == "rect":
        d = _div(case)
        steps = [d[i:i + 3] for i in range(0, len(d), 3)]
        A = _rect_unpack(x[0], case["m"], case["k"], [(a, c) for a, _, c in steps])
        B = _rect_unpack(x[1], case["k"], case["n"], [(c, b) for _, b, c in steps])
        return _rect_pack(A @ B, [(a, b) for a, b, _ in steps])
    if op == "layout":
        return [_pack(x[0].reshape(case["n"], case["n"]).t(), case["n"], case["r"], case["bs"]), x[0]]
    if op == "batched":
        # column-major operands: (A B)^T = B^T A^T on the row-major views
        return [(b.reshape(n, n) @ a.reshape(n, n)).reshape(-1) for (a, b), n in zip(x, _sizes(case))]
    n, r, bs = case["n"], case.get("r", 0), case.get("bs", 1)
    A, B = _unpack(x[0], n, r, bs), _unpack(x[1], n, r, bs)
    if op == "chol":
        P = A @ B.t()
        return _pack(case["alpha"] * _unpack(x[2], n, r, bs) - P if case["alpha"] != 0.0 else -P, n, r, bs)
    return _pack(A @ B, n, r, bs)
