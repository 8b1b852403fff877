"""The device-built problem table of grouped HGEMMs: every entry and tile
descriptor is the words that the host encoder gives."""
import ctypes

import numpy as np
import pytest

import hcblas_b200 as hb

pytestmark = pytest.mark.gpu

ENTRY, MAPS = 512, 384  # bytes of an entry, of its three tensor maps
BN64, AMN, BMN, CTMA = 1, 2, 4, 8

PROBLEM = np.dtype([("a", "u8"), ("b", "u8"), ("c", "u8"), ("lda", "i4"), ("ldb", "i4"),
                    ("ldc", "i4"), ("m", "i4"), ("n", "i4"), ("k", "i4"), ("flags", "i4"),
                    ("pad", "V12")])
assert PROBLEM.itemsize == 64


def up8(v):
    return (v + 7) // 8 * 8


def test_build_matches_encode(handle):
    L = hb.lib()
    i64, vp = ctypes.c_int64, ctypes.c_void_p
    L.hcbk_grouped_encode.argtypes = [vp, ctypes.c_int, ctypes.c_int, i64, i64, i64, vp, i64, vp,
                                      i64, vp, i64]
    L.hcbk_grouped_build.argtypes = [vp, vp, vp, vp, ctypes.c_int, ctypes.c_int, vp]
    pool = hb.DeviceArray(handle, nbytes=1 << 20, dtype=np.uint8)  # addresses only
    rng = np.random.default_rng(0)
    sizes = [1, 7, 8, 16, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 1000, 1024, 2048]
    probs, want, ts, descs = [], [], [0], []
    for i in range(400):
        ta, tb = int(rng.integers(0, 2)), int(rng.integers(0, 2))
        m, n, k = (int(rng.choice(sizes)) for _ in range(3))
        lda = up8(m if ta == 0 else k) + 8 * int(rng.integers(0, 3))
        ldb = up8(k if tb == 0 else n) + 8 * int(rng.integers(0, 3))
        ldc = m if i % 3 else up8(m)
        a, b = (pool.ptr + 16 * int(rng.integers(0, 1000)) for _ in range(2))
        c = pool.ptr + (16 if i % 5 else 2) * int(rng.integers(0, 1000))
        e = (ctypes.c_uint8 * (ENTRY + 128))()
        at = (ctypes.addressof(e) + 127) // 128 * 128
        assert L.hcbk_grouped_encode(at, ta, tb, m, n, k, a, lda, b, ldb, c, ldc) == 0
        w = np.frombuffer((ctypes.c_uint8 * ENTRY).from_address(at), np.uint8).copy()
        tail = w[MAPS:].view(np.int32)
        c_tma = int(tail[11])
        if not c_tma:
            w[256:384] = 0  # the C map is not built
        flags = (BN64 if n <= 64 else 0) | (AMN if ta == 0 else 0) | (BMN if tb else 0) | \
            (CTMA if c_tma else 0)
        probs.append((a, b, c, lda, ldb, ldc, m, n, k, flags, b""))
        want.append(w)
        bn = 64 if n <= 64 else 128
        tm, tn = -(-m // 128), -(-n // bn)
        descs += [(i | flags << 24, t % tm, t // tm, k) for t in range(tm * tn)]
        ts.append(ts[-1] + tm * tn)
    hp, hts = np.array(probs, PROBLEM), np.array(ts, np.int32)
    dp, dts = hb.DeviceArray(handle, hp.view(np.uint8)), hb.DeviceArray(handle, hts)
    for count, on_host in ((len(probs), 0), (256, 1), (1, 1)):  # copied, handed over as parameters
        tiles = ts[count]
        table = hb.DeviceArray(handle, np.zeros(ENTRY * count, np.uint8))
        td = hb.DeviceArray(handle, np.full(4 * tiles + 4, -1, np.int32))
        src = (hp.ctypes.data, hts.ctypes.data) if on_host else (dp.ptr, dts.ptr)
        assert L.hcbk_grouped_build(*src, table.ptr, td.ptr, count, on_host, None) == 0
        got = table.download().reshape(-1, ENTRY)
        for i, w in enumerate(want[:count]):
            assert np.array_equal(got[i, :MAPS], w[:MAPS]), (i, probs[i])
            assert np.array_equal(got[i, MAPS:MAPS + 52], w[MAPS:MAPS + 52]), (i, probs[i])
        d = td.download()
        assert np.array_equal(d[:-4].reshape(-1, 4), np.array(descs[:tiles], np.int64).astype(np.int32))
        assert (d[-4:] == -1).all()


@pytest.mark.parametrize("misaligned", [False, True])
def test_back_to_back_calls_keep_their_order(handle, misaligned):
    """The launches of a pointer-array batch overlap (table builder, grouped
    kernel, the pass over flagged entries): calls queued without a wait between
    them, each reading what the one before wrote, give the words that the same
    calls give one at a time."""
    n, batch, rounds = 96, 40, 12
    rng = np.random.default_rng(3)
    step = n * n + (1 if misaligned else 0)  # every other matrix off 16 bytes
    mats = [hb.DeviceArray(handle, (rng.standard_normal(batch * step + 8) / 16).astype(np.float16))
            for _ in range(3)]
    arrs = [hb.DeviceArray(handle, np.array([m.ptr + 2 * step * i for i in range(batch)], np.uint64))
            for m in mats]
    start = [m.download() for m in mats]

    def play(wait):
        for m, x in zip(mats, start):
            m.upload(x)
        for r in range(rounds):
            a, b, c = (arrs[(r + j) % 3] for j in range(3))
            assert hb.gemm_batched(handle, 0, r & 1, n, n, n, 1.0, a.ptr, n, b.ptr, n, 0.5, c.ptr, n,
                                   batch, np.float16) == 0
            if wait:
                assert hb.device_error(handle) == 0
        return [m.download() for m in mats]

    want = play(True)
    for _ in range(3):
        for g, w in zip(play(False), want):
            assert np.array_equal(g.view(np.uint16), w.view(np.uint16))
    assert hb.device_error(handle) == 0
