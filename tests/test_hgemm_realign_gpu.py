"""HGEMM whose operands or C TMA cannot address (odd leading dimensions, bases
off 16 bytes): the copy into addressable scratch, the transposed product with
its column-wise epilogue, and the calls that keep the CUDA-core kernel."""
import numpy as np
import pytest
import torch

import hcblas_b200 as hb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

U16, U32 = 2.0 ** -11, 2.0 ** -24


def call(h, order, ta, tb, M, N, K, alpha, beta, rng, pad, off):
    ra, ca = (M, K) if ta == "n" else (K, M)
    rb, cb = (K, N) if tb == "n" else (N, K)
    lead = lambda r, c, p: (r if order == O.COL else c) + p
    lines = lambda r, c: c if order == O.COL else r
    lda, ldb, ldc = lead(ra, ca, pad[0]), lead(rb, cb, pad[1]), lead(M, N, pad[2])
    A = rng.standard_normal(lda * lines(ra, ca) + off[0]).astype(np.float16)
    B = rng.standard_normal(ldb * lines(rb, cb) + off[1]).astype(np.float16)
    C = rng.standard_normal(ldc * lines(M, N) + off[2]).astype(np.float16)
    dA, dB, dC = (hb.DeviceArray(h, X) for X in (A, B, C))
    assert hb.lib_gemm(h, order, ta, tb, M, N, K, alpha, dA, lda, dB, ldb, beta, dC, ldc,
                       *off) == 0
    assert hb.device_error(h) == 0
    got, path = dC.download(), hb.hcblasGetLastPath(h)
    op = {"n": 0, "t": 1}
    args = (order, op[ta], op[tb], M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, *off)
    _, ref = O.gemm(*args)
    _, mag = O.gemm(order, op[ta], op[tb], M, N, K, abs(alpha), np.abs(A), lda, np.abs(B), ldb,
                    abs(beta), np.abs(C), ldc, *off)
    err = np.abs(O.view_c(got, order, M, N, ldc, off[2]).astype(np.float64) - ref)
    # one rounding to binary16, and binary32 sums of K + 2 terms (twice: the
    # tensor core truncates where FMA rounds)
    bound = U16 * np.abs(ref) + 2.0 ** -24 + 2 * (K + 2) * U32 * mag
    assert (err <= bound).all(), (path, float((err - bound).max()))
    # nothing outside the M x N window changed
    keep = np.ones(got.size, bool)
    idx = np.arange(lines(M, N))[:, None] * ldc + np.arange(M if order == O.COL else N) + off[2]
    keep[idx.ravel()] = False
    assert np.array_equal(got[keep].view(np.uint16), C[keep].view(np.uint16)), path
    return path


@pytest.mark.parametrize("ta,tb", [("n", "n"), ("n", "t"), ("t", "n"), ("t", "t")])
@pytest.mark.parametrize("M,N,K,beta", [
    (641, 701, 643, 0.0),     # just above the product size that pays for the copy
    (2049, 1027, 129, 0.5),   # tails of one row, one column and one K element
    (8191, 257, 131, -1.0),
    (131, 130, 17001, 0.5),   # one tile of a long K
    (1025, 1031, 1033, 1.0),
])
def test_odd_leading_dimensions(handle, ta, tb, M, N, K, beta):
    rng = np.random.default_rng(M + N + K)
    for order in (O.COL, O.ROW):
        path = call(handle, order, ta, tb, M, N, K, 1.25, beta, rng, (0, 0, 0), (0, 0, 0))
        assert path.startswith("tc.h."), path


@pytest.mark.parametrize("pair", [0, 1, 2])
@pytest.mark.parametrize("pad,off", [
    ((7, 0, 0), (0, 0, 0)),    # A alone off 16 bytes
    ((0, 3, 0), (0, 0, 0)),    # B alone
    ((0, 0, 0), (1, 0, 0)),    # A's base
    ((0, 0, 1), (0, 0, 0)),    # C alone: its columns alternate between even and odd elements
    ((0, 0, 0), (0, 0, 5)),    # C's base
    ((2, 4, 6), (2, 4, 6)),    # 4-byte but not 16-byte aligned
])
def test_alignments(handle, pad, off, pair):
    rng = np.random.default_rng(sum(pad) * 7 + sum(off) + pair)
    assert hb.set_tuning(handle, "tc_pair", pair) == 0
    try:
        for M, N, K, beta in ((512, 1024, 640, 0.0), (1032, 536, 520, 0.75)):
            path = call(handle, O.COL, "n", "t", M, N, K, -0.5, beta, rng, pad, off)
            assert path.startswith("tc.h."), path
    finally:
        hb.set_tuning(handle, "tc_pair", 1)


@pytest.mark.parametrize("M", [130, 136, 1, 7, 9, 127, 129, 255, 257])
def test_c_column_ends(handle, M):
    """Every alignment of a column's two ends, columns shorter than a chunk
    among them (addressable operands, C alone off 16 bytes)."""
    rng = np.random.default_rng(M)
    for ldc_pad in (0, 1, 2, 3):
        for beta in (0.0, 0.5):
            call(handle, O.COL, "t", "n", M, 77, 72, 1.0, beta, rng, (0, 0, ldc_pad), (0, 0, 3))


def test_captured_call_keeps_the_scratch_free_kernel(built_lib):
    """Under the caller's stream capture no scratch may be had: the call is
    accepted as before, on the CUDA cores, and replays correctly; the
    library's own graphs replay the tensor-core form."""
    M = N = K = 801
    rng = np.random.default_rng(5)
    A, B = (rng.standard_normal(M * K).astype(np.float16) for _ in range(2))
    st = torch.cuda.Stream()
    s, h = hb.hcblasCreate(0, st.cuda_stream)
    assert s == 0
    try:
        dA, dB = hb.DeviceArray(h, A), hb.DeviceArray(h, B)
        dC = hb.DeviceArray(h, nbytes=2 * M * N, dtype=np.float16)
        run = lambda: hb.lib_gemm(h, O.COL, "n", "n", M, N, K, 1.0, dA, M, dB, K, 0.0, dC, M)
        assert run() == 0
        assert hb.hcblasGetLastPath(h).startswith("tc.h.")
        eager = dC.download()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            assert run() == 0
            assert hb.hcblasGetLastPath(h).startswith("simt.h.")
        A2 = rng.standard_normal(M * K).astype(np.float16)
        dA.upload(A2)
        g.replay()
        torch.cuda.synchronize()
        _, ref = O.gemm(O.COL, 0, 0, M, N, K, 1.0, A2, M, B, K, 0.0, np.zeros(M * N, np.float16), M)
        got = O.view_c(dC.download(), O.COL, M, N, M).astype(np.float64)
        assert np.linalg.norm(got - ref) <= 2.0 ** -10 * np.linalg.norm(ref)
        assert hb.set_tuning(h, "graphs", 1) == 0
        dA.upload(A)
        for _ in range(3):
            assert run() == 0
        torch.cuda.synchronize()
        assert np.array_equal(dC.download().view(np.uint16), eager.view(np.uint16))
        assert hb.set_tuning(h, "workspace_mb", 1) == 0  # no room for the copies
        assert hb.set_tuning(h, "graphs", 0) == 0
        assert run() == 0
        assert hb.hcblasGetLastPath(h).startswith("simt.h.")
        assert hb.device_error(h) == 0
    finally:
        hb.hcblasDestroy(h)
