"""Native FP64 GEMMs (dmma_gemm.cu) over every cluster split: edges of the
64 x 64 tiles and 16-k slabs, leading dimensions and bases on and off 16
bytes, every op, alpha / beta, batches."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb
from oracle import oracle as O
from tests.test_fma_gemm_gpu import Args

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53


def run(handle, kind, ta, tb, M, N, K, alpha, beta, split, pad=0, off=0, batch=1):
    f = {"d": hb.lib().hcbk_dgemm_dmma, "z": hb.lib().hcbk_zgemm_zmma}[kind]
    f.argtypes = [ctypes.POINTER(Args), ctypes.c_int, ctypes.c_void_p]
    dt = {"d": np.float64, "z": np.complex128}[kind]
    rng = np.random.default_rng(M * 7 + N * 3 + K + 10 * ta + tb)
    mk = lambda n: (rng.standard_normal(n) + (1j * rng.standard_normal(n) if kind == "z" else 0)).astype(dt)
    lda, ldb, ldc = (M if ta == 0 else K) + pad, (K if tb == 0 else N) + pad, M + pad
    sa, sb, sc = lda * (K if ta == 0 else M), ldb * (N if tb == 0 else K), ldc * N
    A, B, C = mk(sa * batch + off), mk(sb * batch + off), mk(sc * batch + off)
    dA, dB, dC = (hb.DeviceArray(handle, X) for X in (A, B, C))
    a = Args(dtype={"d": 1, "z": 3}[kind], op_a=ta, op_b=tb, m=M, n=N, k=K, a=dA.ptr, lda=lda,
             stride_a=sa, a_off=off, b=dB.ptr, ldb=ldb, stride_b=sb, b_off=off, c=dC.ptr, ldc=ldc,
             stride_c=sc, c_off=off, batch=batch, alpha_re=np.real(alpha), alpha_im=np.imag(alpha),
             beta_re=np.real(beta), beta_im=np.imag(beta))
    assert f(ctypes.byref(a), split, None) == 0
    got = dC.download()
    for e in range(batch):
        oa, ob, oc = off + e * sa, off + e * sb, off + e * sc
        _, ref = O.gemm(O.COL, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, oa, ob, oc)
        _, mag = O.gemm(O.COL, min(ta, 1), min(tb, 1), M, N, K, abs(alpha), np.abs(A).real.copy(),
                        lda, np.abs(B).real.copy(), ldb, abs(beta), np.abs(C).real.copy(), ldc,
                        oa, ob, oc)
        err = np.abs(O.view_c(got, O.COL, M, N, ldc, oc) - ref)
        bound = (2 * K + 16) * U64 * np.abs(mag) * 2
        assert (err <= bound).all(), (kind, ta, tb, M, N, K, split, pad, float((err / bound).max()))
    keep = np.ones(got.size, bool)
    for e in range(batch):
        keep[(np.arange(N)[:, None] * ldc + np.arange(M) + off + e * sc).ravel()] = False
    assert np.array_equal(got[keep], C[keep])


@pytest.mark.parametrize("kind,ops", [("d", [(0, 0), (0, 1), (1, 0), (1, 1)]),
                                      ("z", [(0, 0), (0, 2), (2, 0), (2, 2), (1, 2), (1, 1)])])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 16), (65, 63, 17), (63, 130, 48),
                                   (128, 64, 33), (200, 33, 300)])
def test_splits_and_edges(handle, kind, ops, M, N, K):
    for ta, tb in ops:
        for split in (1, 2, 3, 8):
            for pad, off in ((0, 0), (1, 1), (2, 0)):
                run(handle, kind, ta, tb, M, N, K, 1.25, 0.0 if split == 2 else 0.5, split, pad, off)


@pytest.mark.parametrize("kind", "dz")
def test_batches_reuse_the_stages(handle, kind):
    for split in (1, 4):
        run(handle, kind, 0, 1, 70, 130, 100, 0.5 - (0.25j if kind == "z" else 0), 1.0, split, batch=5)
        run(handle, kind, 1, 0, 33, 17, 65, 1.0, 0.0, split, pad=3, batch=4)
