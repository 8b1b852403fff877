"""Autotuner: kernels that share a size bucket keep their own decisions."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("first", ["short", "long"])
def test_kernels_of_one_bucket(tmp_path, first):
    """400 x 400 by K = 130 (short-K kernel) and by K = 256 (K split over a
    cluster) fall into one bucket: whichever is tuned first, the other is tuned
    as well."""
    cache = tmp_path / "tune.txt"
    code = (
        "import sys, numpy as np; sys.path.insert(0, %r)\n"
        "import hcblas_b200 as hb\n"
        "s, h = hb.hcblasCreate(0); hb.set_tuning(h, 'autotune', 1)\n"
        "M = N = 400\n"
        "dA, dB, dC = (hb.DeviceArray(h, np.zeros(M * M, np.float32)) for _ in range(3))\n"
        "for K in %r:\n"
        "    assert hb.lib_gemm(h, hb.ColMajor, 'n', 'n', M, N, K, 1.0, dA, M, dB, K, 0.0, dC, M) == 0\n"
        "    assert ('.k' in hb.hcblasGetLastPath(h)) == (K == 256)\n"
        % (ROOT, (130, 256) if first == "short" else (256, 130)))
    env = dict(os.environ, HCBLAS_AUTOTUNE_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True,
                       timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    keys = [line.rsplit(" ", 1)[0] for line in cache.read_text().splitlines()]
    assert len(keys) == 2 and len(set(keys)) == 2, keys
    assert len({k[k.index("|dt"):] for k in keys}) == 1, keys  # one bucket
