"""HGEMM on copied operands (off 16 bytes): its sums lose no bits against the
CUDA-core kernel, which takes the same call where no scratch may be had."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb
from oracle import oracle as O
from tests.test_fma_gemm_gpu import Args

pytestmark = pytest.mark.gpu


class SimtCfg(ctypes.Structure):  # hcbk_simt_cfg
    _fields_ = [("variant", ctypes.c_int)]


def both(handle, M, N, K, A, B):
    """The product as dispatched, on the CUDA cores, and in binary64."""
    dA, dB = hb.DeviceArray(handle, A), hb.DeviceArray(handle, B)
    dC, dD = (hb.DeviceArray(handle, np.zeros(M * N, np.float16)) for _ in range(2))
    assert hb.lib_gemm(handle, O.COL, "t", "n", M, N, K, 1.0, dA, K, dB, K, 0.0, dC, M) == 0
    assert hb.hcblasGetLastPath(handle).startswith("tc.h.") and hb.device_error(handle) == 0
    f = hb.lib().hcbk_gemm_simt
    f.argtypes = [ctypes.POINTER(Args), SimtCfg, ctypes.c_void_p]
    a = Args(dtype=4, op_a=1, op_b=0, m=M, n=N, k=K, a=dA.ptr, lda=K, b=dB.ptr, ldb=K, c=dD.ptr,
             ldc=M, batch=1, alpha_re=1.0)
    assert f(ctypes.byref(a), SimtCfg(1), None) == 0
    _, ref = O.gemm(O.COL, 1, 0, M, N, K, 1.0, A, K, B, K, 0.0, np.zeros(M * N, np.float16), M)
    return dC.download().reshape(N, M).T, dD.download().reshape(N, M).T, ref


@pytest.mark.parametrize("pair", [1, 2])
@pytest.mark.parametrize("M,N,K", [(2049, 1027, 129), (1025, 777, 777), (515, 519, 4095),
                                   (131, 130, 17001)])
def test_no_more_wrong_roundings_than_the_cuda_cores(handle, M, N, K, pair):
    rng = np.random.default_rng(K)
    A = rng.uniform(-1, 1, M * K).astype(np.float16)
    B = rng.uniform(-1, 1, N * K).astype(np.float16)
    assert hb.set_tuning(handle, "tc_pair", pair) == 0
    try:
        tensor, cuda, ref = both(handle, M, N, K, A, B)
    finally:
        hb.set_tuning(handle, "tc_pair", 1)
    wrong_t, wrong_c = (int((x != ref.astype(np.float16)).sum()) for x in (tensor, cuda))
    # counts of rare events: four standard deviations of the larger one
    assert wrong_t <= wrong_c + 4 * np.sqrt(wrong_c + 1), (wrong_t, wrong_c)


def test_sums_of_one_sign_have_no_bias(handle):
    """Truncated over all of K, sums of one sign come out low by up to 2^-23 of
    their value per 16 K; in chunks of 128 K by at most 8 such steps."""
    M, N, K = 131, 130, 17001
    rng = np.random.default_rng(3)
    A = rng.uniform(0, 1, M * K).astype(np.float16)
    B = rng.uniform(0, 1, N * K).astype(np.float16)
    tensor, _, ref = both(handle, M, N, K, A, B)
    ulp = 2.0 ** (np.floor(np.log2(ref)) - 10)
    bias = float(((tensor.astype(np.float64) - ref) / ulp).mean())
    # 8 x 2^-22 of the value (two units per step) are 2^-8 ulp of binary16 at
    # most; its own rounding has a standard deviation of 0.29 ulp per output
    assert abs(bias) <= 2.0 ** -8 + 4 * 0.29 / np.sqrt(M * N), bias
