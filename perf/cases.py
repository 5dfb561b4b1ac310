"""Performance cases of the emulated FP64 GEMMs: what users of the package ask of it, through its
public calls (oz2.Ozaki2.gemm, zgemm, gemm_grouped and gemm_adaptive), from the smallest call to
the largest.

A case is a dict of plain values. `listed()` gives the cases of record, `draw(rng)` another of the
same ranges; `prepare` makes the inputs and the handle that a program holds before the call, `run`
makes the one call, `work` gives the bytes and operations the call cannot do without, and `exact`
the product as torch computes it in 64 bits.

Kinds:
  gemm      one DGEMM, C = alpha op(A) op(B) + beta C, at a fixed number of moduli s
  zgemm     one ZGEMM (3M form), fixed s
  grouped   many DGEMMs of uneven sizes, ops and s in one call, replayed from a CUDA graph
  adaptive  a batch of DGEMMs of wide dynamic range, the number of moduli chosen per tile

Inputs are column-major, as in BLAS. phi = 0 draws U[-1, 1); phi > 0 draws (u - 0.5) exp(phi g) with
u uniform in [0, 1) and g normal, the wide-range data that needs more moduli.
"""
import math
import os
import random
import sys

import torch

# the package lies in a folder of its own under the working folder, the repository's root
sys.path.insert(0, os.path.join(os.getcwd(), "os2-xe_b200"))
import oz2  # noqa: E402


def _gemm(name, m, n, k, s, ops="NN", alpha=1.0, beta=0.0, pad=0, phi=0.0):
    return {"name": name, "kind": "gemm", "m": m, "n": n, "k": k, "s": s, "ops": ops, "alpha": alpha, "beta": beta,
            "pad": pad, "phi": phi}


def listed():
    return [
        # a single small product inside a larger program: launches and latency, hardly any data
        _gemm("gemm_128", 128, 128, 128, 14),
        # the square product of the workload table's smallest configuration
        _gemm("gemm_1024", 1024, 1024, 1024, 16),
        # the headline DGEMM of the method: large, alpha and beta in use, C padded
        _gemm("gemm_8192", 8192, 8192, 8192, 16, "NN", 1.5, -0.5, 16),
        # few moduli: the fast, low-precision end of the method, both operands transposed
        _gemm("gemm_4096_s8", 4096, 4096, 4096, 8, "TT"),
        # wide-range data, which needs more moduli (more than 62 bits per element)
        _gemm("gemm_wide_s20", 6144, 6144, 6144, 20, "TN", 1.5, -0.5, 16, 4.0),
        # odd sizes and leading dimensions, as an application's own blocking gives them
        _gemm("gemm_ragged", 3001, 1543, 2777, 18, "NT", 1.0, 0.0, 3),
        # the trailing update of a blocked factorisation: short inner dimension, C updated in place
        _gemm("gemm_update", 6000, 6000, 384, 16, "NN", -1.0, 1.0, 0),
        # a long inner dimension, beyond one exact int32 accumulation
        _gemm("gemm_long_k", 1024, 1024, 262144, 16),
        # the complex product, A conjugate-transposed
        {"name": "zgemm_4096", "kind": "zgemm", "m": 4096, "n": 4096, "k": 4096, "s": 16, "ops": "CN", "pad": 8,
         "limit_mb": 0},
        # a ragged complex product under a limit on the workspace
        {"name": "zgemm_ragged", "kind": "zgemm", "m": 3000, "n": 5000, "k": 2000, "s": 16, "ops": "NN", "pad": 0,
         "limit_mb": 4096},
        # 512 uneven problems of a batched application in one graph replay
        {"name": "grouped_512", "kind": "grouped", "count": 512, "lo": 32, "hi": 2048, "s_lo": 14, "s_hi": 20},
        # a batch of the adaptive stream: wide-range problems, s chosen per tile to FP64 accuracy
        {"name": "adaptive_64", "kind": "adaptive", "count": 64, "lo": 256, "hi": 4096, "phi": 8.0, "rows": 40},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "gemm", "gemm_long_k", "zgemm", "grouped", "adaptive"])
    ops = rng.choice("NT") + rng.choice("NT")
    if kind == "gemm":
        m, n, k = (_log_int(rng, 32, 8192) for _ in range(3))
        phi = rng.choice([0.0, 0.0, 1.0, 4.0])
        s = rng.randint(8, 18) if phi == 0.0 else rng.randint(16, 24)
        while m * n * k * s > 8192 ** 3 * 16:
            m = m // 2 + 1
        alpha, beta = rng.choice([(1.0, 0.0), (1.5, -0.5), (-1.0, 1.0)])
        c = _gemm("", m, n, k, s, ops, alpha, beta, rng.choice([0, 1, 8, 16]), phi)
    elif kind == "gemm_long_k":
        m, n = _log_int(rng, 64, 1024), _log_int(rng, 64, 1024)
        c = _gemm("", m, n, _log_int(rng, 16384, 262144), rng.randint(12, 18), ops, 1.0, 0.0, rng.choice([0, 3]))
    elif kind == "zgemm":
        m, n, k = (_log_int(rng, 64, 4096) for _ in range(3))
        c = {"kind": "zgemm", "m": m, "n": n, "k": k, "s": rng.randint(10, 18),
             "ops": rng.choice("NTC") + rng.choice("NTC"), "pad": rng.choice([0, 1, 8]), "limit_mb": 0}
    elif kind == "grouped":
        c = {"kind": "grouped", "count": rng.randint(32, 512), "lo": rng.choice([32, 64, 100]),
             "hi": _log_int(rng, 256, 2048), "s_lo": rng.choice([12, 14, 16]), "s_hi": rng.choice([16, 18, 20])}
    else:
        c = {"kind": "adaptive", "count": rng.randint(8, 64), "lo": 256, "hi": _log_int(rng, 1024, 4096),
             "phi": rng.choice([2.0, 5.0, 8.0]), "rows": rng.choice([0, 20, 40])}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(g, count, phi):
    if phi == 0.0:
        return torch.rand(count, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0
    x = torch.rand(count, dtype=torch.float64, device="cuda", generator=g) - 0.5
    return x.mul_(torch.randn(count, dtype=torch.float64, device="cuda", generator=g).mul_(phi).exp_())


def _stored(op, rows, cols):
    """(stored rows, stored columns) of X with op(X) rows x cols"""
    return (rows, cols) if op == "N" else (cols, rows)


def _gemm_inputs(case, seed):
    """A, B, C as flat column-major buffers and their leading dimensions (complex: pairs)"""
    g = _generator(seed)
    w = 2 if case["kind"] == "zgemm" else 1
    ta, tb = case["ops"]
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    out = []
    for rows, cols in (_stored(ta, m, k), _stored(tb, k, n), (m, n)):
        ld = rows + pad
        out += [_values(g, w * ld * cols, case.get("phi", 0.0)), ld]
    return out


def _group_specs(case, seed):
    """(m, n, k, ops, s) per problem of a grouped case: from the case alone, so that every pass of
    a program that replays its graph sees the same shapes; `seed` gives the data"""
    rnd = random.Random("%d,%d,%d,%d,%d" % tuple(case[x] for x in ("count", "lo", "hi", "s_lo", "s_hi")))
    size = lambda: _log_int(rnd, case["lo"], case["hi"])  # noqa: E731
    return [(size(), size(), size(), rnd.choice("NT") + rnd.choice("NT"), rnd.randint(case["s_lo"], case["s_hi"]))
            for _ in range(case["count"])]


def _group_inputs(case, seed):
    """one arena each for A, B and C, and per problem the views and sizes"""
    specs = _group_specs(case, seed)
    g = _generator(seed)
    A = _values(g, sum(m * k for m, n, k, _, _ in specs), 0.0)
    B = _values(g, sum(k * n for m, n, k, _, _ in specs), 0.0)
    C = torch.zeros(sum(m * n for m, n, k, _, _ in specs), dtype=torch.float64, device="cuda")
    a = b = c = 0
    probs = []
    for m, n, k, ops, s in specs:
        probs.append((m, n, k, ops, s, A[a:a + m * k], B[b:b + k * n], C[c:c + m * n]))
        a, b, c = a + m * k, b + k * n, c + m * n
    return probs, C


def _adaptive_inputs(case, seed):
    """square problems of the adaptive stream: rows of A and columns of B scaled by powers of two"""
    rnd = random.Random("%d,%d,%d,%r,%d" % (case["count"], case["lo"], case["hi"], case["phi"], case["rows"]))
    specs = [(_log_int(rnd, case["lo"], case["hi"]), rnd.uniform(0.0, case["phi"])) for _ in range(case["count"])]
    g = _generator(seed)
    C = torch.zeros(sum(n * n for n, _ in specs), dtype=torch.float64, device="cuda")
    c, r = 0, case["rows"]
    probs = []
    for n, phi in specs:
        mats = []
        for shape in ((1, n), (n, 1)):  # [column][row]: A's rows, B's columns
            e = torch.randint(-r, r + 1, shape, device="cuda", generator=g).double()
            mats.append((_values(g, n * n, max(phi, 1e-3)).view(n, n) * torch.exp2(e)).view(-1))
        probs.append((n, mats[0], mats[1], C[c:c + n * n]))
        c += n * n
    return probs, C


def prepare(case, seed):
    oz = oz2.Ozaki2()
    if case["kind"] == "gemm":
        A, lda, B, ldb, C, ldc = _gemm_inputs(case, seed)
        return {"kind": "gemm", "oz": oz, "out": C,
                "args": (case["ops"][0], case["ops"][1], case["m"], case["n"], case["k"], case["alpha"], A, lda, B, ldb,
                         case["beta"], C, ldc, case["s"])}
    if case["kind"] == "zgemm":
        A, lda, B, ldb, C, ldc = _gemm_inputs(case, seed)
        if case["limit_mb"]:
            oz.set_workspace_limit(case["limit_mb"] << 20)
        return {"kind": "zgemm", "oz": oz, "out": C,
                "args": (case["ops"][0], case["ops"][1], case["m"], case["n"], case["k"], 1.0 + 0.5j, A, lda, B, ldb,
                         0.25 - 0.5j, C, ldc, case["s"])}
    if case["kind"] == "grouped":
        probs, C = _group_inputs(case, seed)
        oz.set_graph_mode(True)
        args = [(ops[0], ops[1], m, n, k, 1.0, A, m if ops[0] == "N" else k, B, k if ops[1] == "N" else n, 0.0, Cv, m, s)
                for m, n, k, ops, s, A, B, Cv in probs]
    else:
        probs, C = _adaptive_inputs(case, seed)
        oz.load_model()
        args = [("N", "N", n, n, n, 1.0, A, n, B, n, 0.0, Cv, n, 16) for n, A, B, Cv in probs]
    return {"kind": case["kind"], "oz": oz, "out": C, "args": args}


# ---------------------------------------------------------------- the call
def run(state):
    oz, kind = state["oz"], state["kind"]
    if kind == "gemm":
        oz.gemm(*state["args"])
    elif kind == "zgemm":
        oz.zgemm(*state["args"])
    elif kind == "grouped":
        oz.gemm_grouped(state["args"])
    else:
        stats = oz.gemm_adaptive(state["args"], 53, oz.ADAPTIVE_MLP)
        return {"C": state["out"], "stats": stats}
    return {"C": state["out"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """bytes: A and B read, C written (and read where beta is not zero). flops: the int8 operations
    of the s products (two per multiply-add; three products per modulus for a ZGEMM), which run at
    twice the bf16 rate; for the adaptive batch those of 16 moduli, about the fewest that carry
    FP64's 53 bits."""
    kind = case["kind"]
    if kind in ("gemm", "zgemm"):
        m, n, k, z = case["m"], case["n"], case["k"], kind == "zgemm"
        old_c = 1 if z or case["beta"] != 0.0 else 0
        return {"bytes": (16 if z else 8) * (m * k + k * n + (1 + old_c) * m * n),
                "flops": (6 if z else 2) * case["s"] * m * n * k}
    if kind == "grouped":
        specs = _group_specs(case, 0)
        return {"bytes": 8 * sum(m * k + k * n + m * n for m, n, k, _, _ in specs),
                "flops": 2 * sum(s * m * n * k for m, n, k, _, s in specs)}
    rnd = random.Random("%d,%d,%d,%r,%d" % (case["count"], case["lo"], case["hi"], case["phi"], case["rows"]))
    sizes = [(_log_int(rnd, case["lo"], case["hi"]), rnd.uniform(0.0, case["phi"]))[0] for _ in range(case["count"])]
    return {"bytes": 24 * sum(n * n for n in sizes), "flops": 2 * 16 * sum(n ** 3 for n in sizes)}


# ---------------------------------------------------------------- 64-bit products by torch
def _op(flat, ld, op, rows, cols):
    """op(X) of a flat column-major buffer as a torch matrix (rows x cols)"""
    r, c = _stored(op, rows, cols)
    X = flat.view(c, ld)[:, :r].t()  # r x c
    return X if op == "N" else (X.t() if op == "T" else X.t().conj())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gemm", "zgemm"):
        A, lda, B, ldb, C, ldc = _gemm_inputs(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        z = kind == "zgemm"
        alpha, beta = (1.0 + 0.5j, 0.25 - 0.5j) if z else (case["alpha"], case["beta"])
        cast = (lambda x: torch.view_as_complex(x.view(-1, 2))) if z else (lambda x: x)
        P = _op(cast(A), lda, case["ops"][0], m, k) @ _op(cast(B), ldb, case["ops"][1], k, n)
        out = cast(C).view(n, ldc)
        out[:, :m] = (alpha * P).t() + (beta * out[:, :m] if beta != 0 else 0.0)
        return {"C": C}
    if kind == "grouped":
        probs, C = _group_inputs(case, seed)
        for m, n, k, ops, s, A, B, Cv in probs:
            P = _op(A, m if ops[0] == "N" else k, ops[0], m, k) @ _op(B, k if ops[1] == "N" else n, ops[1], k, n)
            Cv.view(n, m).copy_(P.t())
        return {"C": C}
    probs, C = _adaptive_inputs(case, seed)
    for n, A, B, Cv in probs:
        torch.matmul(B.view(n, n), A.view(n, n), out=Cv.view(n, n))  # (A B)^T = B^T A^T
    return {"C": C, "stats": None}
