"""Grouped HGEMM calls queued without a wait: each call's table is built on the
GPU in the memory of the last call's, and the product starts while the builder
may still run."""
import numpy as np
import pytest

import hcblas_b200 as hb

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
