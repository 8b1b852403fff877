"""Grouped HGEMM calls queued without a wait: each call's table is built on the
GPU in the memory of the last call's, and the product starts while the builder
may still run.  Entries of the longest lines."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb

from tests.test_grouped_table_gpu import ENTRY, PROBLEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [40, 300])  # handed over as parameters, uploaded
def test_changing_problem_arrays(handle, count):
    """Three arrays in rotation that differ in every field of a problem's entry
    (shape, transposes, leading dimensions, addresses, C by tensor stores or
    not), each call reading what earlier ones wrote: the words that the same
    calls give one at a time."""
    rounds, slot = 12, 160 * 168
    rng = np.random.default_rng(count)
    mats = [hb.DeviceArray(handle, (rng.standard_normal(count * slot) / 16).astype(np.float16))
            for _ in range(3)]
    start = [m.download() for m in mats]
    arrays = []
    for r in range(3):
        probs = []
        for i in range(count):
            m, n, k = (int(v) for v in rng.integers(1, 160, 3))
            ta, tb = (int(v) for v in rng.integers(0, 2, 2))
            lda, ldb = (-(-v // 8) * 8 for v in (m if ta == 0 else k, k if tb == 0 else n))
            if i % 2:
                m = -(-m // 8) * 8
                lda = max(lda, m if ta == 0 else 0)
            a, b, c = (mats[(r + x) % 3].ptr + 2 * slot * i for x in range(3))
            probs.append(hb.GemmProblem(ta, tb, m, n, k, a, lda, b, ldb, c, m))
        arrays.append(probs)

    def play(wait):
        for m, x in zip(mats, start):
            m.upload(x)
        for r in range(rounds):
            assert hb.hgemm_grouped(handle, arrays[r % 3], 1.0, 0.5) == 0
            if wait:
                assert hb.device_error(handle) == 0
        return [m.download().view(np.uint16) for m in mats]

    want = play(True)
    for _ in range(3):
        for g, w in zip(play(False), want):
            assert np.array_equal(g, w)
    assert hb.device_error(handle) == 0


@pytest.mark.parametrize("k", [(1 << 30) - 8, 1 << 30, (1 << 31) - 8])
def test_entries_of_long_lines_match_encode(handle, k):
    """op(A) is one line of k elements: 2 GiB and more of them."""
    L = hb.lib()
    i64, vp = ctypes.c_int64, ctypes.c_void_p
    L.hcbk_grouped_encode.argtypes = [vp, ctypes.c_int, ctypes.c_int, i64, i64, i64, vp, i64, vp,
                                      i64, vp, i64]
    L.hcbk_grouped_build.argtypes = [vp, vp, vp, vp, ctypes.c_int, ctypes.c_int, vp]
    table = hb.DeviceArray(handle, np.zeros(ENTRY, np.uint8))
    desc = hb.DeviceArray(handle, np.zeros(4, np.int32))
    at = 1 << 40  # an address only: nothing is read from it
    e = (ctypes.c_uint8 * (ENTRY + 128))()
    p = (ctypes.addressof(e) + 127) // 128 * 128
    assert L.hcbk_grouped_encode(p, 1, 0, 1, 8, k, at, k, at, k, at + 2, 8) == 0
    want = np.frombuffer((ctypes.c_uint8 * ENTRY).from_address(p), np.uint8)
    prob = np.array([(at, at, at + 2, k, k, 8, 1, 8, k, 1, b"")], PROBLEM)  # 64-wide tiles
    ts = np.array([0, 1], np.int32)
    assert L.hcbk_grouped_build(prob.ctypes.data, ts.ctypes.data, table.ptr, desc.ptr, 1, 1, None) == 0
    assert np.array_equal(table.download()[:256], want[:256])
