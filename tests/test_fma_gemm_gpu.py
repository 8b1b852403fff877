"""The FP32 FMA kernel (fma_gemm.cu) over every tile and cluster split: edges
of its 128- and 64-float tiles and 16-k slabs, ragged leading dimensions,
every op, alpha / beta, and batches; called through the kernel shim so that
sizes the dispatch gives to the short-K kernel run here too."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24


class Args(ctypes.Structure):  # hcbk_gemm_args
    _fields_ = [("dtype", ctypes.c_int), ("op_a", ctypes.c_int), ("op_b", ctypes.c_int)] + \
        [(n, ctypes.c_int64) for n in ("m", "n", "k")] + \
        [f for x in "abc" for f in ((x, ctypes.c_void_p), ("ld" + x, ctypes.c_int64),
                                    ("stride_" + x, ctypes.c_int64), (x + "_off", ctypes.c_int64))] + \
        [(x + "_array", ctypes.c_void_p) for x in "abc"] + \
        [("batch", ctypes.c_int64), ("select", ctypes.c_void_p)] + \
        [(n, ctypes.c_double) for n in ("alpha_re", "alpha_im", "beta_re", "beta_im")]


class Cfg(ctypes.Structure):
    _fields_ = [("tile", ctypes.c_int), ("split", ctypes.c_int)]


def run(handle, kind, ta, tb, M, N, K, alpha, beta, tile, split, pad=0, off=0, batch=1):
    f = hb.lib().hcbk_gemm_f32
    f.argtypes = [ctypes.POINTER(Args), Cfg, ctypes.c_void_p]
    dt = {"s": np.float32, "c": np.complex64}[kind]
    rng = np.random.default_rng(M * 7 + N * 3 + K + 10 * ta + tb)
    mk = lambda n: (rng.standard_normal(n) + (1j * rng.standard_normal(n) if kind == "c" else 0)).astype(dt)
    lda, ldb, ldc = (M if ta == 0 else K) + pad, (K if tb == 0 else N) + pad, M + pad
    sa, sb, sc = lda * (K if ta == 0 else M), ldb * (N if tb == 0 else K), ldc * N
    A, B, C = mk(sa * batch + off), mk(sb * batch + off), mk(sc * batch + off)
    dA, dB, dC = (hb.DeviceArray(handle, X) for X in (A, B, C))
    a = Args(dtype={"s": 0, "c": 2}[kind], op_a=ta, op_b=tb, m=M, n=N, k=K, a=dA.ptr, lda=lda,
             stride_a=sa, a_off=off, b=dB.ptr, ldb=ldb, stride_b=sb, b_off=off, c=dC.ptr, ldc=ldc,
             stride_c=sc, c_off=off, batch=batch, alpha_re=np.real(alpha), alpha_im=np.imag(alpha),
             beta_re=np.real(beta), beta_im=np.imag(beta))
    assert f(ctypes.byref(a), Cfg(tile, split), None) == 0
    got = dC.download()
    for e in range(batch):
        oa, ob, oc = off + e * sa, off + e * sb, off + e * sc
        _, ref = O.gemm(O.COL, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, oa, ob, oc)
        _, mag = O.gemm(O.COL, min(ta, 1), min(tb, 1), M, N, K, abs(alpha), np.abs(A).real.astype(np.float32),
                        lda, np.abs(B).real.astype(np.float32), ldb, abs(beta),
                        np.abs(C).real.astype(np.float32), ldc, oa, ob, oc)
        err = np.abs(O.view_c(got, O.COL, M, N, ldc, oc) - ref)
        # sums of K products (2 K real ones), split at most eight ways, alpha and beta
        bound = (2 * K + 16) * U32 * np.abs(mag) * 2
        assert (err <= bound).all(), (kind, ta, tb, M, N, K, tile, split, pad, float((err / bound).max()))
    keep = np.ones(got.size, bool)
    for e in range(batch):
        keep[(np.arange(N)[:, None] * ldc + np.arange(M) + off + e * sc).ravel()] = False
    assert np.array_equal(got[keep], C[keep])


@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("kind,ops", [("s", [(0, 0), (0, 1), (1, 0), (1, 1)]),
                                      ("c", [(0, 0), (0, 2), (2, 0), (2, 2), (1, 2), (1, 1)])])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 16), (65, 63, 17), (127, 130, 48),
                                   (128, 256, 129), (200, 33, 300)])
def test_tiles_splits_and_edges(handle, tile, kind, ops, M, N, K):
    for ta, tb in ops:
        for split in (1, 2, 3, 8):
            for pad, off in ((0, 0), (1, 1), (4, 0)):
                beta = 0.0 if split == 2 else 0.5
                run(handle, kind, ta, tb, M, N, K, 1.25, beta, tile, split, pad, off)


@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("kind", "sc")
def test_batches_reuse_the_stages(handle, tile, kind):
    for split in (1, 4):
        run(handle, kind, 0, 1, 70, 130, 100, 0.5 - (0.25j if kind == "c" else 0), 1.0, tile, split,
            batch=5)
        run(handle, kind, 1, 0, 33, 17, 65, 1.0, 0.0, tile, split, pad=3, batch=4)


def test_integers_are_exact_whatever_the_split(handle):
    """Sums of integers below 2^24: the same words from every tile and split
    (the dispatch's choices among them)."""
    M, N, K = 150, 90, 2000
    rng = np.random.default_rng(1)
    A = rng.integers(-8, 9, M * K).astype(np.float32)
    B = rng.integers(-8, 9, N * K).astype(np.float32)
    dA, dB = hb.DeviceArray(handle, A), hb.DeviceArray(handle, B)
    dC = hb.DeviceArray(handle, nbytes=4 * M * N, dtype=np.float32)
    assert hb.lib_gemm(handle, O.COL, "n", "t", M, N, K, 1.0, dA, M, dB, N, 0.0, dC, M) == 0
    assert ".k" in hb.hcblasGetLastPath(handle)
    exp = (A.reshape(K, M).T.astype(np.float64) @ B.reshape(K, N)).T.ravel()
    assert np.array_equal(dC.download(), exp)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_stay_in_their_row(handle, bad):
    M, N, K = 130, 70, 40
    rng = np.random.default_rng(2)
    A = rng.standard_normal(M * K).astype(np.float32)
    B = np.abs(rng.standard_normal(N * K)).astype(np.float32) + 1
    A[5 + 3 * M] = bad  # op(A)(5, 3)
    dA, dB = hb.DeviceArray(handle, A), hb.DeviceArray(handle, B)
    dC = hb.DeviceArray(handle, np.full(M * N, np.nan, np.float32))
    assert hb.lib_gemm(handle, O.COL, "n", "t", M, N, K, 1.0, dA, M, dB, N, 0.0, dC, M) == 0
    got = dC.download().reshape(N, M).T
    assert np.isfinite(np.delete(got, 5, 0)).all()
    assert np.isnan(got[5]).all() if np.isnan(bad) else (got[5] == bad).all()
