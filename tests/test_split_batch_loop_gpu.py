"""Split-K kernels (fma_gemm.cu, dmma_gemm.cu) whose batch exceeds the grid's
65535 rows of blocks: a block then takes several entries, and its shared memory
passes from one entry's sums to the next entry's slabs.  Integers, so that
every word is known."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb
from oracle import oracle as O
from tests.test_fma_gemm_gpu import Args, Cfg

pytestmark = pytest.mark.gpu

GRID_Y = 65535
TYPES = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}


def integers(rng, n, kind):
    x = rng.integers(-8, 9, n).astype(np.float64)
    if kind in "cz":
        x = x + 1j * rng.integers(-8, 9, n)
    return x.astype(TYPES[kind])


def check(got, C, beta, products, a_of, b_of, M, N, K):
    """Every entry against its integer product (batch x N x M); entries on
    either side of the turn against the oracle as well."""
    batch = len(products)
    exp = products + np.asarray(beta, C.dtype) * C.reshape(batch, N, M)
    bad = np.flatnonzero((got.reshape(batch, -1) != exp.reshape(batch, -1)).any(1))
    assert bad.size == 0, (C.dtype, bad[:10])
    for e in list(range(8)) + list(range(GRID_Y, GRID_Y + 24)):
        w = slice(e * M * N, (e + 1) * M * N)
        out, _ = O.gemm(O.COL, 0, 0, M, N, K, 1.0, a_of(e), M, b_of(e), K, beta, C[w], M)
        assert np.array_equal(out, got[w]), (C.dtype, e)


@pytest.mark.parametrize("kind", "sdcz")
@pytest.mark.parametrize("M,N", [(8, 1), (33, 2)])
def test_blocks_with_several_entries(handle, kind, M, N):
    """Through the kernel shim: every split, both FP32 tiles; the entries' B
    are overlapping windows one element apart."""
    f = {"s": hb.lib().hcbk_gemm_f32, "c": hb.lib().hcbk_gemm_f32, "d": hb.lib().hcbk_dgemm_dmma,
         "z": hb.lib().hcbk_zgemm_zmma}[kind]
    single = kind in "sc"
    f.argtypes = [ctypes.POINTER(Args), Cfg if single else ctypes.c_int, ctypes.c_void_p]
    batch = GRID_Y + 70
    rng = np.random.default_rng(M + N)
    for split in (1, 2, 8):
        K = 16 * split + 21
        A, B = integers(rng, M * K, kind), integers(rng, batch + K * N, kind)
        C = integers(rng, M * N * batch, kind)
        for tile in ((0, 1) if single else (0,)):
            dA, dB, dC = (hb.DeviceArray(handle, X) for X in (A, B, C))
            a = Args(dtype="sdcz".index(kind), op_a=0, op_b=0, m=M, n=N, k=K, a=dA.ptr, lda=M,
                     stride_a=0, b=dB.ptr, ldb=K, stride_b=1, c=dC.ptr, ldc=M, stride_c=M * N,
                     batch=batch, alpha_re=1.0, beta_re=1.0)
            assert f(ctypes.byref(a), Cfg(tile, split) if single else split, None) == 0
            win = np.lib.stride_tricks.sliding_window_view(B, K * N)[:batch].reshape(batch, N, K)
            check(dC.download(), C, 1.0, win @ A.reshape(K, M), lambda e: A,
                  lambda e: B[e:e + K * N], M, N, K)


@pytest.mark.parametrize("kind,K,batch", [("s", 20480, 66017), ("d", 32768, 65721)])
def test_pointer_array_batch_that_the_plan_splits(handle, kind, K, batch):
    """The same through the public entry point: pointers that name a few
    operands, at a batch for which the plan shares each tile's K."""
    M = N = 8
    rng = np.random.default_rng(K)
    A, B = integers(rng, 2 * M * K, kind), integers(rng, 3 * K * N, kind)
    C = integers(rng, M * N * batch, kind)
    dA, dB, dC = (hb.DeviceArray(handle, X) for X in (A, B, C))
    esz = A.itemsize
    ptrs = [np.array([d.ptr + esz * step * (e % some) for e in range(batch)], np.uint64)
            for d, step, some in ((dA, M * K, 2), (dB, K * N, 3), (dC, M * N, batch))]
    pA, pB, pC = (hb.DeviceArray(handle, p) for p in ptrs)
    if kind == "d":
        plan = hb.lib().hcbk_gemm_f64_split
        plan.argtypes = [ctypes.c_int] + [ctypes.c_int64] * 4
        assert plan(0, M, N, K, batch) == 2
    assert hb.gemm_batched(handle, hb.HCBLAS_OP_N, hb.HCBLAS_OP_N, M, N, K, 1.0, pA.ptr, M, pB.ptr,
                           K, 0.5, pC.ptr, M, batch, TYPES[kind]) == 0
    if kind == "s":
        assert hb.hcblasGetLastPath(handle).endswith(".k2")
    a, b = A.reshape(2, K, M), B.reshape(3, N, K)
    pairs = np.stack([b[e % 3] @ a[e % 2] for e in range(6)])
    check(dC.download(), C, 0.5, pairs[np.arange(batch) % 6], lambda e: a[e % 2], lambda e: b[e % 3],
          M, N, K)
