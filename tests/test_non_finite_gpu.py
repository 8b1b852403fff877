"""Infinities and NaN in the kernels of long products: the FP32 and FP64 split-K
kernels over whole and split K, and the HGEMM epilogues by columns."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb
from tests.test_fma_gemm_gpu import Args, Cfg

pytestmark = pytest.mark.gpu

TYPES = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("kind", "sdcz")
def test_bad_values_stay_in_their_row(handle, kind, bad):
    """op(A)(5, 3) is bad, op(B) positive: row 5 is bad, all others are finite;
    C is full of NaN and beta 0.  K ends inside a slab."""
    f = {"s": hb.lib().hcbk_gemm_f32, "c": hb.lib().hcbk_gemm_f32, "d": hb.lib().hcbk_dgemm_dmma,
         "z": hb.lib().hcbk_zgemm_zmma}[kind]
    single, cplx = kind in "sc", kind in "cz"
    f.argtypes = [ctypes.POINTER(Args), Cfg if single else ctypes.c_int, ctypes.c_void_p]
    M, N, K = 130, 70, 601
    rng = np.random.default_rng(2)
    mk = lambda *s: (rng.uniform(1, 2, s) + (1j * rng.uniform(1, 2, s) if cplx else 0)).astype(TYPES[kind])
    for ta, tb in ((0, 1), (1, 0)) + (((2, 2),) if cplx else ()):
        A, B = mk(K, M) if ta == 0 else mk(M, K), mk(N, K) if tb == 0 else mk(K, N)
        A[(3, 5) if ta == 0 else (5, 3)] = bad  # complex: imaginary part 0
        dA, dB = hb.DeviceArray(handle, A.ravel()), hb.DeviceArray(handle, B.ravel())
        for tile in (0, 1) if single else (0,):
            for split in (1, 2, 8):
                dC = hb.DeviceArray(handle, np.full(M * N, np.nan, TYPES[kind]))
                a = Args(dtype="sdcz".index(kind), op_a=ta, op_b=tb, m=M, n=N, k=K, a=dA.ptr,
                         lda=A.shape[1], b=dB.ptr, ldb=B.shape[1], c=dC.ptr, ldc=M, batch=1,
                         alpha_re=1.0)
                assert f(ctypes.byref(a), Cfg(tile, split) if single else split, None) == 0
                got = dC.download().reshape(N, M).T
                assert np.isfinite(np.delete(got, 5, 0)).all(), (ta, tb, tile, split)
                if cplx:  # alpha's imaginary part, 0, times an infinity is NaN
                    assert not (np.isfinite(got[5].real) | np.isfinite(got[5].imag)).any()
                else:
                    assert np.isnan(got[5]).all() if np.isnan(bad) else (got[5] == bad).all()


@pytest.mark.parametrize("pair", [0, 1, 2])
@pytest.mark.parametrize("M,N,K,off16", [(801, 803, 805, True), (2049, 1027, 129, True),
                                         (8191, 257, 136, False), (131, 1032, 1040, False)])
def test_c_is_not_read_when_beta_is_zero(handle, M, N, K, off16, pair):
    """Columns off 16 bytes (copied operands, or C alone): C full of NaN, which
    stays between the columns."""
    rng = np.random.default_rng(M)
    ld = K if off16 else -(-K // 8) * 8
    A, B = (rng.integers(-1, 2, r * ld).astype(np.float16) for r in (M, N))
    C = np.full((N, M + 2), np.nan, np.float16)
    dA, dB, dC = (hb.DeviceArray(handle, x.ravel()) for x in (A, B, C))
    assert hb.set_tuning(handle, "tc_pair", pair) == 0
    try:
        assert hb.lib_gemm(handle, hb.ColMajor, "t", "n", M, N, K, 1.0, dA, ld, dB, ld, 0.0, dC,
                           M + 2) == 0
        assert hb.hcblasGetLastPath(handle).startswith("tc.h.")
    finally:
        hb.set_tuning(handle, "tc_pair", 1)
    got = dC.download().reshape(N, M + 2)
    a, b = (x.reshape(-1, ld)[:, :K].astype(np.float32) for x in (A, B))
    assert np.array_equal(got[:, :M], (b @ a.T).astype(np.float16))
    assert np.isnan(got[:, M:]).all()
