"""SGEMM with an operand off 16 bytes, large enough for its copy into
addressable [k][mn] lines: every pair of transposes, either operand alone,
tails of the 32 x 32 blocks, and the same sums when the operands are read in
place."""
import numpy as np
import pytest
import torch  # noqa: F401  (creates the CUDA context the handles share)

import hcblas_b200 as hb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24
COPY = "pack.realign_f32"


def run(order, ta, tb, M, N, K, beta, pad, off, limit_mb):
    rng = np.random.default_rng(M + N + K)
    ra, ca = (M, K) if ta == "n" else (K, M)
    rb, cb = (K, N) if tb == "n" else (N, K)
    lead = lambda r, c, p: (r if order == O.COL else c) + p
    lines = lambda r, c: c if order == O.COL else r
    lda, ldb, ldc = lead(ra, ca, pad[0]), lead(rb, cb, pad[1]), lead(M, N, pad[2])
    A = rng.standard_normal(lda * lines(ra, ca) + off[0]).astype(np.float32)
    B = rng.standard_normal(ldb * lines(rb, cb) + off[1]).astype(np.float32)
    C = rng.standard_normal(ldc * lines(M, N) + off[2]).astype(np.float32)
    status, h = hb.hcblasCreate()
    assert status == 0
    try:
        if limit_mb:
            hb.set_tuning(h, "workspace_mb", limit_mb)
        hb.set_profiling(h, True)
        dA, dB, dC = (hb.DeviceArray(h, X) for X in (A, B, C))
        assert hb.lib_gemm(h, order, ta, tb, M, N, K, 1.25, dA, lda, dB, ldb, beta, dC, ldc,
                           *off) == 0
        got = dC.download()
        copied = COPY in hb.get_profile(h)
    finally:
        hb.hcblasDestroy(h)
    return got, copied, (order, ta, tb, A, lda, B, ldb, C, ldc)


@pytest.mark.parametrize("M,N,K,beta,pad,off", [
    (2049, 2047, 2045, 0.5, (0, 0, 0), (0, 0, 0)),  # one and 31 of 32 in the last blocks
    (2048, 2080, 2048, 0.0, (1, 0, 0), (0, 0, 0)),  # A alone
    (2080, 2048, 2048, -1.0, (0, 0, 0), (0, 3, 0)),  # B's base alone
])
@pytest.mark.parametrize("ta,tb", [("n", "n"), ("n", "t"), ("t", "n"), ("t", "t")])
def test_copied_operands(ta, tb, M, N, K, beta, pad, off):
    for order in (O.COL, O.ROW):
        args = (order, ta, tb, M, N, K, beta, pad, off)
        got, copied, (_, _, _, A, lda, B, ldb, C, ldc) = run(*args, 0)
        assert copied
        # 16 columns against the oracle in 64 bits: K + 2 roundings
        cols = np.linspace(0, N - 1, 16).astype(int)
        v = lambda X, r, c, ld, o: np.lib.stride_tricks.as_strided(
            X[o:], (r, c), (4, 4 * ld) if order == O.COL else (4 * ld, 4))
        a = v(A, *((M, K) if ta == "n" else (K, M)), lda, off[0]).astype(np.float64)
        b = v(B, *((K, N) if tb == "n" else (N, K)), ldb, off[1]).astype(np.float64)
        a = a if ta == "n" else a.T
        b = (b if tb == "n" else b.T)[:, cols]
        c0 = v(C, M, N, ldc, off[2])[:, cols].astype(np.float64)
        c1 = v(got, M, N, ldc, off[2])[:, cols].astype(np.float64)
        ref = 1.25 * (a @ b) + beta * c0
        mag = 1.25 * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c0)
        assert (np.abs(c1 - ref) <= (K + 2) * U32 * mag).all()
        # 1 MiB of workspace: the operands are read where they are
        place, copied, _ = run(*args, 1)
        assert not copied
        d = np.abs(v(place, M, N, ldc, off[2])[:, cols].astype(np.float64) - ref)
        assert (d <= (K + 2) * U32 * mag).all()
