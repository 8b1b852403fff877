"""The scratch of calls that copy their operands: its limit under the graphs
knob, streams that do not wait for one another, and captures on other streams."""
import numpy as np
import pytest
import torch

import hcblas_b200 as hb

pytestmark = pytest.mark.gpu


class Product:
    """An HGEMM with odd leading dimensions (integers: every word is known)."""

    def __init__(self, seed, M=801, N=803, K=805):
        rng = np.random.default_rng(seed)
        self.shape = M, N, K
        self.a, self.b = (rng.integers(-2, 3, s).astype(np.float16) for s in ((K, M), (N, K)))
        self.want = (self.b.astype(np.float64) @ self.a).astype(np.float16)

    def upload(self, h):
        self.d = [hb.DeviceArray(h, x.ravel()) for x in (self.a, self.b, np.zeros_like(self.want))]

    def run(self, h):
        M, N, K = self.shape
        return hb.lib_gemm(h, hb.ColMajor, "n", "n", M, N, K, 1.0, self.d[0], M, self.d[1], K, 0.0,
                           self.d[2], M)

    def check(self):
        torch.cuda.synchronize()
        assert np.array_equal(self.d[2].download().reshape(self.want.shape), self.want)


@pytest.fixture
def stream_handle(built_lib):
    st = torch.cuda.Stream()
    s, h = hb.hcblasCreate(0, st.cuda_stream)
    assert s == 0
    yield h, st
    hb.hcblasDestroy(h)


@pytest.mark.parametrize("limits", [(0, 1, 0), (1, 0, 1)])
def test_changed_limit_holds_for_repeated_calls(stream_handle, limits):
    h, _ = stream_handle
    assert hb.set_tuning(h, "graphs", 1) == 0
    p = Product(1)
    p.upload(h)
    for limit in limits:
        assert hb.set_tuning(h, "workspace_mb", limit) == 0
        for _ in range(3):
            assert p.run(h) == 0
            assert hb.hcblasGetLastPath(h).startswith("simt.h." if limit else "tc.h."), limit
        p.check()


def test_streams_do_not_wait_for_one_another(stream_handle):
    """Scratch that a call on one stream has handed back is not taken on another
    by waiting for the first."""
    h, one = stream_handle
    two = torch.cuda.Stream()
    p, q = Product(2), Product(3)
    p.upload(h)
    q.upload(h)
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    busy, done = torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(one):
        torch.cuda._sleep(4_000_000_000)  # about two seconds
    assert p.run(h) == 0
    busy.record(one)
    assert hb.hcblasSetStream(h, two.cuda_stream) == 0
    assert q.run(h) == 0
    done.record(two)
    done.synchronize()
    assert not busy.query()
    hb.hcblasSetStream(h, one.cuda_stream)
    p.check()
    q.check()


def test_capture_on_another_stream_goes_on(stream_handle):
    """A handle's first call that copies its operands, while this thread captures
    another stream in global mode: neither disturbs the other."""
    h, _ = stream_handle
    p = Product(4)
    p.upload(h)
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
        x.add_(1)
        assert p.run(h) == 0
        x.add_(1)
    g.replay()
    p.check()
    assert (x == 2).all()


@pytest.mark.parametrize("M,N,K,copies", [
    (3400, 24, 40001, 2), (24, 3400, 40001, 2), (3400, 3401, 40001, 4),  # 3354 lines fit
    (131, 130, 600001, 1), (300, 24, 1000001, 3),  # 223, 134 lines fit
])
@pytest.mark.parametrize("ta,tb", [("n", "t"), ("t", "n")])
def test_copies_above_the_cap_go_in_panels(handle, M, N, K, copies, ta, tb):
    """Either operand has half of the scratch, 256 MiB."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)

    class Dev:
        dtype = np.dtype(np.float16)

        def __init__(self, rows, cols):
            self.t = torch.randint(-2, 3, (rows, cols), generator=gen, device="cuda").half()
            self.ptr = self.t.data_ptr()

    a = Dev(K, M + 1) if ta == "n" else Dev(M, K)  # lines of the column-major operands
    b = Dev(N, K) if tb == "n" else Dev(K, N + 1)
    c = Dev(N, M + 3)
    want = c.t.clone()
    A = a.t[:, :M].T if ta == "n" else a.t
    B = b.t if tb == "n" else b.t[:, :N].T
    prod = torch.zeros(N, M, device="cuda", dtype=torch.float64)
    for k in range(0, K, 4096):  # exact: sums of integers
        prod += B[:, k:k + 4096].double() @ A[:, k:k + 4096].double().T
    want[:, :M] = (prod + 0.5 * c.t[:, :M].double()).half()
    torch.cuda.synchronize()
    hb.set_profiling(handle, True)
    try:
        assert hb.lib_gemm(handle, hb.ColMajor, ta, tb, M, N, K, 1.0, a, a.t.shape[1], b,
                           b.t.shape[1], 0.5, c, M + 3) == 0
        launches = hb.get_profile(handle)["pack.realign_f16"][0]
    finally:
        hb.set_profiling(handle, False)
    assert hb.device_error(handle) == 0
    assert launches == copies
    assert torch.equal(c.t, want)
