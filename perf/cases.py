"""The GEMM work whose speed this repository watches.

A case is one call of the library's C ABI (through the ctypes binding) as a
program makes it: operands in device memory, host scalars, a handle that the
program keeps.  ``prepare`` makes the operands and binds the arguments, ``run``
makes the call, ``exact`` gives the same result in binary64 from torch alone.

Kinds of case:

* ``gemm``     one ``hcblasLib{S,D,C,Z,H}gemm`` call (the class method's C shim:
               both storage orders).
* ``batch``    ``hcblas{S,D,C,Z,H}gemmBatched`` over device-resident pointer
               arrays, the batched entry point of the reference.
* ``grouped``  ``hcblas{H,S}gemmGrouped`` over problems of uneven shapes.

The handles live as long as the process, one per math mode, as in a program that
creates its handles at start-up; the operands change from state to state.
"""
import ctypes
import math
import random

import numpy as np
import torch

import hcblas_b200 as hb

_NP = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128, "h": np.float16}
_TORCH = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128,
          "h": torch.float16}
_SIZE = {"s": 4, "d": 8, "c": 8, "z": 16, "h": 2}
_OPS = {"N": hb.HCBLAS_OP_N, "T": hb.HCBLAS_OP_T, "C": hb.HCBLAS_OP_C}
#: (math mode, its count) of each named mode; 0 leaves the count to the accuracy target
_MODES = {"native": (hb.HCBLAS_MATH_NATIVE, 0), "split": (hb.HCBLAS_MATH_SPLIT_BF16, 6),
          "crt": (hb.HCBLAS_MATH_OZAKI_CRT, 0)}
_handles = {}


def _gemm(name, dtype, ops, m, n, k, alpha=1.0, beta=0.0, order="col", mode="native",
          alpha_im=0.0, beta_im=0.0):
    return {"name": name, "kind": "gemm", "dtype": dtype, "mode": mode, "order": order, "ops": ops,
            "m": m, "n": n, "k": k, "alpha": alpha, "alpha_im": alpha_im, "beta": beta,
            "beta_im": beta_im}


def listed():
    return [
        # the reference tests' smallest ordinary product: one call's latency
        _gemm("sgemm_tiny", "s", "NN", 189, 9, 19, 1.0, 1.0),
        # an ordinary square product of a row-major program
        _gemm("sgemm_rowmajor_1024", "s", "NN", 1024, 1024, 1024, 1.0, 0.5, order="row"),
        # few outputs from a long reduction: a weight gradient or a Gram block
        _gemm("sgemm_long_k", "s", "NT", 777, 1133, 14522, 1.0, 1.0),
        # a large product with dimensions as they come: leading dimensions off 16 bytes
        _gemm("sgemm_ragged_large", "s", "TN", 8378, 8378, 1133),
        # a rank-256 update of a large matrix on the split-BF16 tensor-core mode
        _gemm("sgemm_split_update", "s", "TN", 8192, 8192, 256, 1.0, 1.0, mode="split"),
        # binary64 on the native path, a tall panel with odd dimensions
        _gemm("dgemm_ragged", "d", "NN", 8378, 777, 1133, 1.0, 0.5),
        # binary64 at native accuracy on the int8 tensor cores: the headline product
        _gemm("dgemm_crt_4096", "d", "NT", 4096, 4096, 4096, mode="crt"),
        # a large binary16 product, aligned as a trained model's layers are
        _gemm("hgemm_8192", "h", "NN", 8192, 8192, 8192),
        # binary16 with odd dimensions: a vocabulary or a feature count as it comes
        _gemm("hgemm_ragged", "h", "TN", 8378, 1133, 777, 1.0, 0.5),
        # many small equal products at once, each its own allocation (attention heads)
        {"name": "hgemm_batch_512x128", "kind": "batch", "dtype": "h", "ops": "NN", "m": 128,
         "n": 128, "k": 128, "count": 512, "alpha": 1.0, "beta": 0.0},
        # many small products of uneven shapes at once (experts, blocks of a sparse matrix)
        {"name": "hgemm_grouped_4096", "kind": "grouped", "dtype": "h", "count": 4096, "low": 16,
         "high": 1024, "alpha": 1.0, "beta": 0.0},
        # complex binary32 with the left operand conjugated (correlation, beam forming)
        _gemm("cgemm_cn_2048", "c", "CN", 2048, 2048, 2048, 1.0, 0.5, alpha_im=0.5, beta_im=-0.25),
    ]


def _between(rng, low, high):
    """An integer whose logarithm is uniform; a multiple of 8 half of the time."""
    v = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return max(low, min(high, (v + 4) // 8 * 8 if v >= 16 and rng.random() < 0.5 else v))


def draw(rng: random.Random):
    kind = rng.choice(["gemm"] * 7 + ["batch", "grouped"])
    if kind == "batch":
        m, n, k = (_between(rng, 8, 256) for _ in range(3))
        return {"kind": "batch", "dtype": rng.choice("hhsd"), "ops": rng.choice(["NN", "NT", "TN", "TT"]),
                "m": m, "n": n, "k": k, "count": _between(rng, 8, 512), "alpha": 1.0,
                "beta": rng.choice([0.0, 0.5])}
    if kind == "grouped":
        low = _between(rng, 8, 64)
        return {"kind": "grouped", "dtype": rng.choice("hs"), "count": _between(rng, 16, 4096),
                "low": low, "high": _between(rng, 2 * low, 1024), "alpha": 1.0, "beta": 0.0}
    dtype, mode = rng.choice([("s", "native"), ("s", "native"), ("s", "split"), ("d", "native"),
                              ("d", "crt"), ("c", "native"), ("z", "native"), ("h", "native"),
                              ("h", "native")])
    most = 1.1e12 if dtype == "h" else 1.5e11
    low = 256 if mode != "native" else 8
    while True:
        m, n = _between(rng, low, 8378), _between(rng, low, 8378)
        k = _between(rng, low, 14522)
        if (8 if dtype in "cz" else 2) * m * n * k <= most:
            break
    return {"kind": "gemm", "dtype": dtype, "mode": mode, "order": rng.choice(["col", "col", "row"]),
            "ops": rng.choice(["NN", "NT", "TN", "TT"] + (["CN", "NC"] if dtype in "cz" else [])),
            "m": m, "n": n, "k": k, "alpha": 1.0, "alpha_im": 0.0,
            "beta": rng.choice([0.0, 0.0, 0.5, 1.0]), "beta_im": 0.0}


# ------------------------------------------------------------------- inputs --


def _uniform(gen, count, dtype):
    """U[-1, 1) in the storage type."""
    real = {"c": torch.float32, "z": torch.float64}.get(dtype, _TORCH[dtype])
    lanes = 2 if dtype in "cz" else 1
    v = torch.rand(count * lanes, generator=gen, device="cuda", dtype=real).mul_(2).sub_(1)
    return torch.view_as_complex(v.view(-1, 2)) if lanes == 2 else v


def _normal(gen, count, dtype):
    """N(0, 1) in the storage type (real and imaginary parts for complex)."""
    real = {"c": torch.float32, "z": torch.float64}.get(dtype, _TORCH[dtype])
    lanes = 2 if dtype in "cz" else 1
    v = torch.randn(count * lanes, generator=gen, device="cuda", dtype=real)
    return torch.view_as_complex(v.view(-1, 2)) if lanes == 2 else v


def _stored(rows, cols, op, order):
    """(rows, columns, leading dimension) of the stored operand of op(X) = rows x cols."""
    r, c = (rows, cols) if op == "N" else (cols, rows)
    return r, c, (r if order == "col" else c)


def _gemm_inputs(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    m, n, k, dt = case["m"], case["n"], case["k"], case["dtype"]
    return _normal(gen, m * k, dt), _normal(gen, k * n, dt), _normal(gen, m * n, dt)


def _batch_inputs(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    m, n, k, b, dt = case["m"], case["n"], case["k"], case["count"], case["dtype"]
    # each matrix starts on a 256-byte boundary, as separate allocations do
    up = 256 // _SIZE[dt]
    pa, pb, pc = (-(-v // up) * up for v in (m * k, k * n, m * n))
    return (_uniform(gen, b * pa, dt), pa), (_uniform(gen, b * pb, dt), pb), (_uniform(gen, b * pc, dt), pc)


def _grouped_problems(case, seed):
    """Shapes, ops, leading dimensions and element offsets of every problem: the
    shapes follow from the case alone, so that every seed has the same work."""
    rng = np.random.default_rng([case["count"], case["low"], case["high"]])
    half = case["dtype"] == "h"
    up = 128 if half else 64  # matrices on 256-byte boundaries
    probs, at = [], [0, 0, 0]
    for _ in range(case["count"]):
        ta, tb = int(rng.integers(0, 2)), int(rng.integers(0, 2))
        m, n, k = (int(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"] + 1))))
                   for _ in range(3))
        # binary16 operands are stored with columns on 16-byte boundaries
        r8 = (lambda v: -(-v // 8) * 8) if half else (lambda v: v)
        lda, ldb = r8(k if ta else m), r8(n if tb else k)
        sizes = (lda * (m if ta else k), ldb * (k if tb else n), m * n)
        probs.append((ta, tb, m, n, k, lda, ldb, m, *at))
        at = [a + -(-s // up) * up for a, s in zip(at, sizes)]
    return probs, at


def _grouped_inputs(case, seed, probs, at):
    gen = torch.Generator("cuda").manual_seed(seed)
    return (_uniform(gen, at[0], case["dtype"]), _uniform(gen, at[1], case["dtype"]),
            _uniform(gen, at[2], case["dtype"]))


# --------------------------------------------------------------------- calls --


def _handle(mode):
    if mode not in _handles:
        status, h = hb.hcblasCreate(0)
        assert status == hb.HCBLAS_STATUS_SUCCESS, status
        if mode != "native":
            assert hb.hcblasSetMathMode(h, *_MODES[mode]) == 0
        if mode == "crt":
            assert hb.hcblasSetAccuracyTarget(h, hb.HCBLAS_ACCURACY_NATIVE) == 0
        _handles[mode] = h
    return _handles[mode]


def _scalars(case):
    dt = np.dtype(_NP[case["dtype"]])
    cplx = case["dtype"] in "cz"
    alpha = complex(case["alpha"], case.get("alpha_im", 0.0)) if cplx else case["alpha"]
    beta = complex(case["beta"], case.get("beta_im", 0.0)) if cplx else case["beta"]
    return alpha, beta, hb.scalar_bytes(dt, alpha), hb.scalar_bytes(dt, beta)


def prepare(case, seed):
    L, p = hb.lib(), case["dtype"].upper()
    alpha, beta, al, be = _scalars(case)
    m, n, k = (case.get(d) for d in "mnk")
    if case["kind"] == "gemm":
        h = _handle(case["mode"])
        A, B, C = _gemm_inputs(case, seed)
        ops, order = case["ops"], case["order"]
        lda = _stored(m, k, ops[0], order)[2]
        ldb = _stored(k, n, ops[1], order)[2]
        ldc = m if order == "col" else n
        ta, tb = ops[0].lower().encode(), ops[1].lower().encode()
        o = hb.ColMajor if order == "col" else hb.RowMajor
        a, b, c = A.data_ptr(), B.data_ptr(), C.data_ptr()
        if case["dtype"] in "cz":
            args = (h, o, ta, tb, m, n, k, al.ctypes.data, a, 0, lda, b, 0, ldb, be.ctypes.data, c,
                    0, ldc)
        else:
            args = (h, o, ta, tb, m, n, k, al.ctypes.data, a, lda, b, ldb, be.ctypes.data, c, ldc,
                    0, 0, 0)
        return {"call": getattr(L, f"hcblasLib{p}gemm"), "args": args, "out": C,
                "keep": (A, B, al, be)}
    h = _handle("native")
    if case["kind"] == "batch":
        pools = _batch_inputs(case, seed)
        arrays = []
        for x, pitch in pools:
            step = pitch * _SIZE[case["dtype"]]
            arrays.append(x.data_ptr() + step * torch.arange(case["count"], device="cuda",
                                                             dtype=torch.int64))
        ops = case["ops"]
        lda, ldb = _stored(m, k, ops[0], "col")[2], _stored(k, n, ops[1], "col")[2]
        args = (h, _OPS[ops[0]], _OPS[ops[1]], m, n, k, al.ctypes.data, arrays[0].data_ptr(), lda,
                arrays[1].data_ptr(), ldb, be.ctypes.data, arrays[2].data_ptr(), m, case["count"])
        return {"call": getattr(L, f"hcblas{p}gemmBatched"), "args": args, "out": pools[2][0],
                "keep": (pools, arrays, al, be)}
    probs, at = _grouped_problems(case, seed)
    A, B, C = _grouped_inputs(case, seed, probs, at)
    size = _SIZE[case["dtype"]]
    a, b, c = A.data_ptr(), B.data_ptr(), C.data_ptr()
    table = (hb.GemmProblem * len(probs))(*(
        (ta, tb, mm, nn, kk, a + size * ao, lda, b + size * bo, ldb, c + size * co, ldc)
        for ta, tb, mm, nn, kk, lda, ldb, ldc, ao, bo, co in probs))
    args = (h, len(probs), ctypes.cast(table, ctypes.c_void_p), al.ctypes.data, be.ctypes.data)
    return {"call": getattr(L, f"hcblas{p}gemmGrouped"), "args": args, "out": C,
            "keep": (A, B, table, al, be)}


def run(state):
    status = state["call"](*state["args"])
    if status != 0:
        raise RuntimeError(f"the call returned {status}")
    return state["out"]


# ---------------------------------------------------------------------- work --


def work(case):
    size = _SIZE[case["dtype"]]
    reads_c = 2 if case["beta"] or case.get("beta_im") else 1
    if case["kind"] == "grouped":
        probs, _ = _grouped_problems(case, 0)
        mnk = [(p[2], p[3], p[4]) for p in probs]
    else:
        mnk = [(case["m"], case["n"], case["k"])] * case.get("count", 1)
    return {"bytes": size * sum(m * k + k * n + reads_c * m * n for m, n, k in mnk),
            "flops": (8 if case["dtype"] in "cz" else 2) * sum(m * n * k for m, n, k in mnk)}


# --------------------------------------------------------------------- exact --


def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _opped(x, rows, cols, op, order, ld=None):
    """op(X) as a rows x cols matrix in 64 bits, from its flat storage."""
    r, c, natural = _stored(rows, cols, op, order)
    ld = ld or natural
    v = _wide(x[:ld * (c if order == "col" else r)].view(-1, ld)[:, :(r if order == "col" else c)])
    v = v.t() if order == "col" else v
    return v if op == "N" else v.t() if op == "T" else v.conj().t()


def exact(case, seed):
    alpha, beta, _, _ = _scalars(case)
    m, n, k = (case.get(d) for d in "mnk")
    if case["kind"] == "gemm":
        A, B, C = _gemm_inputs(case, seed)
        ops, order = case["ops"], case["order"]
        r = alpha * (_opped(A, m, k, ops[0], order) @ _opped(B, k, n, ops[1], order))
        r += beta * _opped(C, m, n, "N", order)
        return (r.t() if order == "col" else r).contiguous().view(-1)
    if case["kind"] == "batch":
        (A, pa), (B, pb), (C, pc) = _batch_inputs(case, seed)
        out = _wide(C)
        for i in range(case["count"]):
            r = alpha * (_opped(A[i * pa:], m, k, case["ops"][0], "col") @
                         _opped(B[i * pb:], k, n, case["ops"][1], "col"))
            c = out[i * pc:i * pc + m * n]
            c.copy_((r.t() + beta * c.view(n, m)).reshape(-1))
        return out
    probs, at = _grouped_problems(case, seed)
    A, B, C = _grouped_inputs(case, seed, probs, at)
    out = _wide(C)
    for ta, tb, m, n, k, lda, ldb, ldc, ao, bo, co in probs:
        r = alpha * (_opped(A[ao:], m, k, "NT"[ta], "col", lda) @
                     _opped(B[bo:], k, n, "NT"[tb], "col", ldb))
        c = out[co:co + m * n]
        c.copy_((r.t() + beta * c.view(n, m)).reshape(-1))
    return out
