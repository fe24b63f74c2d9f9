"""The calls whose speed this library is kept to, as a user's program makes them on one GPU.

Each case is a dict of plain values.  `prepare` makes what such a program holds before the call (device operands in
column-major storage, a grouped plan where there is one), `run` makes one call of the library's public entry points
on torch's current stream, `work` states the bytes and operations the call cannot do without, and `exact` its
results in float64 from torch alone.  A column-major matrix with leading dimension ld is a torch tensor of shape
(columns, ld): element (i, j) is t[j, i].
"""
import ctypes as C
import math

import numpy as np
import torch

import mojoblas_b200 as mb
from mojoblas_b200 import _lib as L

MODES = {"plain": mb.PLAIN, "bf16x3": mb.BF16X3, "bf16x6": mb.BF16X6, "ozaki": mb.OZAKI}
DTYPES = {"f32": torch.float32, "f64": torch.float64}
SLICES = 7  # the default of the library's routines: meets plain FP64's error


def _gemm(dtype, mode, ta, tb, m, n, k, alpha=1.0, beta=0.0, **more):
    return dict(op="gemm", dtype=dtype, mode=mode, ta=ta, tb=tb, m=m, n=n, k=k, alpha=alpha, beta=beta, **more)


def listed():
    return [
        # the smallest calls, in the drop-in precision: launch latency and a chip that one wave does not fill.
        # A layer-sized product with both scalars, and an odd-sized float64 one of a host application's inner loop
        _gemm("f32", "plain", "N", "N", 512, 512, 512, 1.5, 0.5, name="sgemm_plain_nn_512"),
        _gemm("f64", "plain", "T", "N", 300, 521, 257, name="dgemm_plain_tn_300x521x257"),
        # the drop-in precision at a size that fills the chip
        _gemm("f32", "plain", "N", "T", 4096, 4096, 4096, name="sgemm_plain_nt_4096"),
        # split-precision products: the largest call, and an ordinary one with ragged, unaligned sizes
        _gemm("f32", "bf16x6", "N", "T", 8192, 8192, 8192, name="sgemm_bf16x6_nt_8192"),
        _gemm("f32", "bf16x6", "T", "N", 1531, 1023, 2047, name="sgemm_bf16x6_tn_1531x1023x2047"),
        # float64 work of a solver: the product and the triangular solve with many right-hand sides
        _gemm("f64", "ozaki", "N", "N", 4096, 4096, 4096, name="dgemm_ozaki_nn_4096"),
        dict(op="trsm", dtype="f64", mode="ozaki", side="L", uplo="L", ta="N", diag="N", m=4096, n=4096,
             name="dtrsm_ozaki_llnn_4096"),
        # a Gram (covariance) matrix from tall data
        dict(op="syrk", dtype="f32", mode="bf16x6", uplo="L", ta="N", n=8192, k=2048, name="ssyrk_bf16x6_ln_8192x2048"),
        # thousands of small problems of uneven sizes in one plan: products and triangular solves
        dict(op="grouped_gemm", mode="bf16x6", ta="N", tb="N", count=4096, lo=16, hi=512, sizes_seed=41,
             name="grouped_sgemm_bf16x6_4096"),
        dict(op="grouped_trsm", uplo="L", ta="N", diag="N", count=2048, lo=8, hi=256, max_rhs=64, sizes_seed=42,
             name="grouped_strsm_2048"),
        # reverse mode: both gradients of a product, both gradients of a triangular solve
        dict(op="gemm_adjoint", mode="bf16x6", ta="N", tb="N", m=3072, n=2048, k=1024,
             name="sgemm_adjoint_bf16x6_3072x2048x1024"),
        dict(op="trsm_adjoint", mode="bf16x6", side="L", uplo="L", ta="N", diag="N", m=2048, n=512,
             name="strsm_adjoint_bf16x6_2048x512"),
    ]


def draw(rng):
    """A case of the same ranges: each family as often as the list has it, sizes log-uniform, half of them odd as they
    fall and half multiples of 32 (what padded data has)."""
    def size(lo, hi):
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return v if rng.random() < 0.5 else max(lo, v // 32 * 32)

    def nt():
        return rng.choice("NT")

    def scalars():
        return dict(alpha=1.0, beta=0.0) if rng.random() < 0.5 else dict(alpha=1.5, beta=0.5)

    kind = rng.choice(["small32", "small64", "plain", "split", "split", "ozaki", "trsm", "syrk", "grouped_gemm",
                       "grouped_trsm", "gemm_adjoint", "trsm_adjoint"])
    if kind == "small32":
        return _gemm("f32", "plain", nt(), nt(), size(64, 1024), size(64, 1024), size(64, 1024), **scalars())
    if kind == "small64":
        return _gemm("f64", "plain", nt(), nt(), size(64, 1024), size(64, 1024), size(64, 1024), **scalars())
    if kind == "plain":
        return _gemm("f32", "plain", nt(), nt(), size(1024, 4096), size(1024, 4096), size(512, 4096), **scalars())
    if kind == "split":
        return _gemm("f32", rng.choice(["bf16x3", "bf16x6", "bf16x6"]), nt(), nt(), size(512, 8192), size(512, 8192),
                     size(256, 8192), **scalars())
    if kind == "ozaki":
        return _gemm("f64", "ozaki", nt(), nt(), size(512, 4096), size(512, 4096), size(512, 4096), **scalars())
    if kind == "trsm":
        return dict(op="trsm", dtype="f64", mode="ozaki", side=rng.choice("LR"), uplo=rng.choice("LU"), ta=nt(),
                    diag="N", m=size(1024, 4096), n=size(1024, 4096))
    if kind == "syrk":
        return dict(op="syrk", dtype="f32", mode="bf16x6", uplo=rng.choice("LU"), ta=nt(), n=size(1024, 8192),
                    k=size(256, 2048))
    if kind == "grouped_gemm":
        return dict(op="grouped_gemm", mode=rng.choice(["plain", "bf16x6", "bf16x6"]), ta=nt(), tb=nt(),
                    count=size(256, 4096), lo=16, hi=rng.choice([128, 256, 512]), sizes_seed=rng.randrange(1 << 30))
    if kind == "grouped_trsm":
        return dict(op="grouped_trsm", uplo=rng.choice("LU"), ta=nt(), diag="N", count=size(256, 2048), lo=8,
                    hi=rng.choice([64, 128, 256]), max_rhs=rng.choice([16, 64]), sizes_seed=rng.randrange(1 << 30))
    if kind == "gemm_adjoint":
        return dict(op="gemm_adjoint", mode="bf16x6", ta=nt(), tb=nt(), m=size(512, 4096), n=size(512, 4096),
                    k=size(512, 4096))
    return dict(op="trsm_adjoint", mode="bf16x6", side=rng.choice("LR"), uplo=rng.choice("LU"), ta=nt(), diag="N",
                m=size(512, 2048), n=size(512, 2048))


# ---- inputs ------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, cols, ld, dtype=torch.float32):
    return torch.rand((cols, ld), generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _normal(g, cols, ld, dtype=torch.float32):
    return torch.randn((cols, ld), generator=g, device="cuda", dtype=dtype)


def _triangle(g, order, dtype):
    """A well-conditioned triangular system's matrix, both triangles filled: N(0, 1) / sqrt(order) beside a dominant
    diagonal."""
    a = _normal(g, order, order, dtype).div_(math.sqrt(order))
    a.diagonal().copy_(order + _normal(g, 1, order, dtype)[0].abs())
    return a


def _ch(c):
    return c.encode()


def _check(status, what):
    if status != 0:
        raise mb.MbgError(what, status)


def _log_uniform(rng, lo, hi, count):
    return np.clip(np.round(np.exp(rng.uniform(np.log(lo), np.log(hi), count))), lo, hi).astype(np.int64)


def _grouped_sizes(case):
    """Per problem: m, n, k of a product; the order and the right-hand sides of a solve."""
    rng = np.random.default_rng(case["sizes_seed"])
    if case["op"] == "grouped_gemm":
        return tuple(_log_uniform(rng, case["lo"], case["hi"], case["count"]) for _ in range(3))
    return _log_uniform(rng, case["lo"], case["hi"], case["count"]), rng.integers(1, case["max_rhs"] + 1, case["count"])


def _pack(sizes):
    """Offsets of matrices of `sizes` elements in one buffer, each on a 256-byte boundary as an allocator places
    them, and the buffer's length."""
    padded = (np.asarray(sizes) + 63) // 64 * 64
    ends = np.cumsum(padded)
    return ends - padded, int(ends[-1])


def _grouped_gemm_layout(case):
    m, n, k = _grouped_sizes(case)
    return (m, n, k), _pack(m * k), _pack(k * n), _pack(m * n)


def _grouped_trsm_layout(case):
    order, rhs = _grouped_sizes(case)
    return (order, rhs), _pack(order * order), _pack(order * rhs)


def _inputs(case, seed):
    g, op = _generator(seed), case["op"]
    if op == "gemm":
        dt = DTYPES[case["dtype"]]
        m, n, k = case["m"], case["n"], case["k"]
        s = {"a": _uniform(g, *((k, m) if case["ta"] == "N" else (m, k)), dt),
             "b": _uniform(g, *((n, k) if case["tb"] == "N" else (k, n)), dt)}
        if case["beta"] != 0:
            s["c0"] = _uniform(g, n, m, dt)
        return s
    if op == "trsm":
        dt = DTYPES[case["dtype"]]
        return {"a": _triangle(g, case["m"] if case["side"] == "L" else case["n"], dt),
                "b0": _normal(g, case["n"], case["m"], dt)}
    if op == "syrk":
        return {"a": _uniform(g, *((case["k"], case["n"]) if case["ta"] == "N" else (case["n"], case["k"])))}
    if op == "grouped_gemm":
        _, (_, na), (_, nb), _ = _grouped_gemm_layout(case)
        return {"a": _uniform(g, 1, na)[0], "b": _uniform(g, 1, nb)[0]}
    if op == "grouped_trsm":
        (order, _), (oa, na), (_, nb) = _grouped_trsm_layout(case)
        a = _normal(g, 1, na)[0]
        padded = torch.from_numpy(np.diff(np.append(oa, na))).cuda()
        a.div_(torch.repeat_interleave(torch.from_numpy(np.sqrt(order)).float().cuda(), padded))
        at = np.concatenate([o + np.arange(v) * (v + 1) for o, v in zip(oa, order)])
        diagonal = torch.from_numpy(np.repeat(order, order)).float().cuda()
        a[torch.from_numpy(at).cuda()] = diagonal + _normal(g, 1, len(at))[0].abs()
        return {"a": a, "b0": _normal(g, 1, nb)[0]}
    if op == "gemm_adjoint":
        m, n, k = case["m"], case["n"], case["k"]
        return {"a": _uniform(g, *((k, m) if case["ta"] == "N" else (m, k))),
                "b": _uniform(g, *((n, k) if case["tb"] == "N" else (k, n))), "g": _normal(g, n, m)}
    # the adjoint of a solve has its solution X at hand: op(A) X = B (X op(A) = B) with B ~ N(0, 1)
    m, n = case["m"], case["n"]
    a = _triangle(g, m if case["side"] == "L" else n, torch.float32)
    b = _normal(g, n, m)
    return {"a": a, "x": _solve(case, a, b, case["ta"]).float().contiguous(), "g": _normal(g, n, m)}


class Plan:
    """A grouped plan with the buffers its problems point into, as a program keeps it between calls."""

    def __init__(self, create, mode, problems):
        self.problems, self.handle = problems, C.c_void_p()
        _check(create(mode, len(problems), problems, C.byref(self.handle)), "grouped plan")

    def execute(self):
        _check(L.load().mbg_plan_execute(self.handle), "plan_execute")

    def __del__(self):
        if self.handle:
            L.load().mbg_plan_destroy(self.handle)


def prepare(case, seed):
    lib = mb.load()
    mb.set_stream(torch.cuda.current_stream())  # device operands: calls are enqueued on torch's stream
    mb.set_sync(False)
    s, op = _inputs(case, seed), case["op"]
    s["case"] = case
    if op == "gemm":
        s["c"] = torch.zeros((case["n"], case["m"]), device="cuda", dtype=DTYPES[case["dtype"]])
    elif op == "trsm":
        s["x"] = torch.zeros_like(s["b0"])
    elif op == "syrk":
        s["c"] = torch.zeros((case["n"], case["n"]), device="cuda")
    elif op == "grouped_gemm":
        (m, n, k), (oa, _), (ob, _), (oc, nc) = _grouped_gemm_layout(case)
        s["c"] = torch.zeros(nc, device="cuda")
        pa, pb, pc = s["a"].data_ptr(), s["b"].data_ptr(), s["c"].data_ptr()
        ta, tb = _ch(case["ta"]), _ch(case["tb"])
        problems = (L.SgemmProblem * case["count"])()
        for i in range(case["count"]):
            mi, ni, ki = int(m[i]), int(n[i]), int(k[i])
            problems[i] = L.SgemmProblem(ta, tb, mi, ni, ki, 1.0, 0.0, pa + 4 * int(oa[i]), mi if ta == b"N" else ki,
                                         pb + 4 * int(ob[i]), ki if tb == b"N" else ni, pc + 4 * int(oc[i]), mi)
        s["plan"] = Plan(lib.mbg_sgemm_grouped_plan, MODES[case["mode"]], problems)
    elif op == "grouped_trsm":
        (order, rhs), (oa, _), (ob, _) = _grouped_trsm_layout(case)
        s["x"] = torch.zeros_like(s["b0"])
        pa, px = s["a"].data_ptr(), s["x"].data_ptr()
        problems = (L.StrsmProblem * case["count"])()
        for i in range(case["count"]):
            v = int(order[i])
            problems[i] = L.StrsmProblem(b"L", _ch(case["uplo"]), _ch(case["ta"]), _ch(case["diag"]), v, int(rhs[i]),
                                         1.0, pa + 4 * int(oa[i]), v, px + 4 * int(ob[i]), v)
        s["plan"] = Plan(lib.mbg_strsm_grouped_plan, mb.PLAIN, problems)
    elif op == "gemm_adjoint":
        s["da"], s["db"] = torch.zeros_like(s["a"]), torch.zeros_like(s["b"])
    else:
        s["da"], s["db"] = torch.zeros_like(s["a"]), torch.zeros_like(s["g"])
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "gemm":
        if case["beta"] != 0:
            s["c"].copy_(s["c0"])  # C is updated in place
        mb.gemm(case["ta"], case["tb"], case["m"], case["n"], case["k"], case["alpha"], s["a"], s["a"].shape[1],
                s["b"], s["b"].shape[1], case["beta"], s["c"], case["m"], mode=MODES[case["mode"]], slices=SLICES)
        return s["c"]
    if op == "trsm":
        s["x"].copy_(s["b0"])  # X overwrites B
        mb.trsm(case["side"], case["uplo"], case["ta"], case["diag"], case["m"], case["n"], 1.0, s["a"],
                s["a"].shape[1], s["x"], case["m"], mode=MODES[case["mode"]], slices=SLICES)
        return s["x"]
    if op == "syrk":
        mb.syrk(case["uplo"], case["ta"], case["n"], case["k"], 1.0, s["a"], s["a"].shape[1], 0.0, s["c"], case["n"],
                mode=MODES[case["mode"]])
        return s["c"]
    if op == "grouped_gemm":
        s["plan"].execute()
        return s["c"]
    if op == "grouped_trsm":
        s["x"].copy_(s["b0"])
        s["plan"].execute()
        return s["x"]
    lib, mode = L.load(), MODES[case["mode"]]
    if op == "gemm_adjoint":
        _check(lib.mbg_sgemm_adjoint(mode, _ch(case["ta"]), _ch(case["tb"]), case["m"], case["n"], case["k"], 1.0,
                                     s["a"].data_ptr(), s["a"].shape[1], s["b"].data_ptr(), s["b"].shape[1],
                                     s["g"].data_ptr(), case["m"], s["da"].data_ptr(), s["da"].shape[1],
                                     s["db"].data_ptr(), s["db"].shape[1]), "sgemm_adjoint")
    else:
        _check(lib.mbg_strsm_adjoint(mode, _ch(case["side"]), _ch(case["uplo"]), _ch(case["ta"]), _ch(case["diag"]),
                                     case["m"], case["n"], 1.0, s["a"].data_ptr(), s["a"].shape[1],
                                     s["x"].data_ptr(), case["m"], s["g"].data_ptr(), case["m"], s["db"].data_ptr(),
                                     case["m"], s["da"].data_ptr(), s["da"].shape[1]), "strsm_adjoint")
    return {"da": s["da"], "db": s["db"]}


# ---- what a call cannot do without ---------------------------------------------------------------------------

def work(case):
    op = case["op"]
    size = 8 if case.get("dtype") == "f64" else 4
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": size * (m * k + k * n + m * n * (1 if case["beta"] == 0 else 2)), "flops": 2 * m * n * k}
    if op == "trsm":
        m, n = case["m"], case["n"]
        t = m if case["side"] == "L" else n
        return {"bytes": size * (t * (t + 1) // 2 + 2 * m * n), "flops": m * n * t}
    if op == "syrk":
        n, k = case["n"], case["k"]
        return {"bytes": size * (n * k + n * (n + 1) // 2), "flops": n * (n + 1) * k}
    if op == "grouped_gemm":
        m, n, k = _grouped_sizes(case)
        return {"bytes": int(size * (m * k + k * n + m * n).sum()), "flops": int(2 * (m * n * k).sum())}
    if op == "grouped_trsm":
        order, rhs = _grouped_sizes(case)
        return {"bytes": int(size * (order * (order + 1) // 2 + 2 * order * rhs).sum()),
                "flops": int((order * order * rhs).sum())}
    if op == "gemm_adjoint":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": size * (2 * m * k + 2 * k * n + m * n), "flops": 4 * m * n * k}
    m, n = case["m"], case["n"]
    t, r = (m, n) if case["side"] == "L" else (n, m)
    return {"bytes": size * (t * (t + 1) + 3 * m * n), "flops": 2 * t * t * r}  # the solve and one triangle of W X^T


# ---- the results in float64 ----------------------------------------------------------------------------------

def _op(t, trans):
    """op(M) as an ordinary float64 matrix, of a column-major M."""
    return (t.T if trans == "N" else t).double()


def _solve(case, a, b, trans, flip=False):
    """op(A) X = B or X op(A) = B in float64, column-major in and out; `flip` for op(A)^T in the place of op(A)."""
    full = a.double().T  # M(i, j) = a[j, i]
    full = torch.tril(full) if case["uplo"] == "L" else torch.triu(full)
    t = full if (trans == "N") != flip else full.T
    upper = (case["uplo"] == "U") == ((trans == "N") != flip)
    bb = b.double().T
    if case["side"] == "L":
        x = torch.linalg.solve_triangular(t, bb, upper=upper)
    else:
        x = torch.linalg.solve_triangular(t, bb, upper=upper, left=False)
    return x.T


def exact(case, seed):
    s, op = _inputs(case, seed), case["op"]
    if op == "gemm":
        c = torch.mm(_op(s["a"], case["ta"]), _op(s["b"], case["tb"])).mul_(case["alpha"])
        if case["beta"] != 0:
            c += case["beta"] * s["c0"].double().T
        return c.T
    if op == "trsm":
        return _solve(case, s["a"], s["b0"], case["ta"])
    if op == "syrk":
        a = _op(s["a"], case["ta"])
        c = torch.mm(a, a.T)
        return (torch.tril(c) if case["uplo"] == "L" else torch.triu(c)).T
    if op == "grouped_gemm":
        (m, n, k), (oa, _), (ob, _), (oc, nc) = _grouped_gemm_layout(case)
        c = torch.zeros(nc, device="cuda", dtype=torch.float64)
        for i in range(case["count"]):
            mi, ni, ki = int(m[i]), int(n[i]), int(k[i])
            a = s["a"][oa[i]:oa[i] + mi * ki].view((ki, mi) if case["ta"] == "N" else (mi, ki))
            b = s["b"][ob[i]:ob[i] + ki * ni].view((ni, ki) if case["tb"] == "N" else (ki, ni))
            c[oc[i]:oc[i] + mi * ni] = torch.mm(_op(a, case["ta"]), _op(b, case["tb"])).T.reshape(-1)
        return c
    if op == "grouped_trsm":
        (order, rhs), (oa, _), (ob, nb) = _grouped_trsm_layout(case)
        x = s["b0"].double()  # what lies between the problems stays
        for i in range(case["count"]):
            v, r = int(order[i]), int(rhs[i])
            a, b = s["a"][oa[i]:oa[i] + v * v].view(v, v), s["b0"][ob[i]:ob[i] + v * r].view(r, v)
            x[ob[i]:ob[i] + v * r] = _solve(dict(case, side="L"), a, b, case["ta"]).reshape(-1)
        return x
    if op == "gemm_adjoint":
        a, b, g = _op(s["a"], case["ta"]), _op(s["b"], case["tb"]), s["g"].double().T
        da, db = torch.mm(g, b.T), torch.mm(a.T, g)  # of op(A) and op(B)
        return {"da": da.T if case["ta"] == "N" else da, "db": db.T if case["tb"] == "N" else db}
    w = _solve(case, s["a"], s["g"], case["ta"], flip=True).T
    x = s["x"].double().T
    # d op(A) = -W X^T on the left, -X^T W on the right; A's own gradient is its transpose where op transposes
    da = -(torch.mm(w, x.T) if case["side"] == "L" else torch.mm(x.T, w))
    da = da if case["ta"] == "N" else da.T
    return {"da": (torch.tril(da) if case["uplo"] == "L" else torch.triu(da)).T, "db": w.T}
