"""The host-buffer drop-ins on both sides of the size from which they cut a
call into groups of chunks, pageable and pinned, and what the grouped path
reports of damaged streams.  Streams, sums and floats are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu
EB = float(np.float32(2e-4))


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    Z.lib()
    return t


def wave(n, f):
    rng = np.random.default_rng(n)
    x = np.sin(np.arange(n, dtype=np.float32) * np.float32(f))
    x[: n // 2] += rng.normal(0, 0.01, n // 2).astype(np.float32)
    return x


@pytest.mark.parametrize("n,T", [((1 << 24) - 1, 16), (1 << 24, 2), ((1 << 24) + 9, 16), ((3 << 23) + 5, 7)])
def test_grouped_and_whole(torch, port, n, T):
    L = 32
    x, y = wave(n, 1e-3), wave(n, 7e-4)
    sx, sy = port.compress(x, EB, L, T), port.compress(y, EB, L, T)
    dx, sxy = port.decompress(sx, n, EB, L, T).view(np.uint32), port.homadd(sx, sy, n, EB, L, T)
    Z.set_omp_threads(T)
    cap = 4 * n + 8 * T + 4096
    for pinned in (False, True):
        def host(count, dtype):
            return torch.zeros(count, dtype=dtype, pin_memory=pinned).numpy()
        xh, hs = host(n, torch.float32), host(cap, torch.uint8)
        xh[:] = x
        size = Z.ZCCL_float_openmp_threadblock_arg(hs, xh, 0, EB, n, L)
        assert hs[:size].tobytes() == sx
        Z.ZCCL_float_decompress_openmp_threadblock_arg(xh, n, EB, L, hs)
        assert np.array_equal(xh.view(np.uint32), dx)
        acc, sep = host(cap, torch.uint8), host(cap, torch.uint8)
        acc[: len(sy)] = np.frombuffer(sy, np.uint8)
        total = Z.ZCCL_float_homomophic_add_openmp_threadblock(sep, 0, n, EB, L, hs, acc)
        assert total == len(sxy) and sep[:total].tobytes() == sxy
        total = Z.ZCCL_float_homomophic_add_openmp_threadblock(acc, 0, n, EB, L, hs, acc)
        assert total == len(sxy) and acc[:total].tobytes() == sxy


def test_grouped_path_reports_bad_streams(torch, port):
    n, L, T = 1 << 25, 32, 16  # four groups
    good = port.compress(wave(n, 1e-3), EB, L, T)
    Z.set_omp_threads(T)
    hdr = np.frombuffer(good[: 8 * T], "<u8")
    out = np.zeros(n, np.float32)

    def host(b):
        h = np.zeros(4 * n + 8 * T + 4096, np.uint8)
        h[: len(b)] = np.frombuffer(b, np.uint8)
        return h

    bad, far = host(good), host(good)
    bad[8 * T + int(hdr[6]) + 64:][:32] = 0xEE  # inside chunk 6, no width bytes
    far[8 * 5: 8 * 6] = np.frombuffer(np.uint64(3 * far.size).tobytes(), np.uint8)  # chunk 5 starts past the end
    for h in (bad, far):
        with pytest.raises(Z.ZcclError):
            Z.ZCCL_float_decompress_openmp_threadblock_arg(out, n, EB, L, h)
    acc = host(good)
    with pytest.raises(Z.ZcclError):
        Z.ZCCL_float_homomophic_add_openmp_threadblock(acc, 0, n, EB, L, bad, acc)
    acc = host(good)
    total = Z.ZCCL_float_homomophic_add_openmp_threadblock(acc, 0, n, EB, L, host(good), acc)
    assert acc[:total].tobytes() == port.homadd(good, good, n, EB, L, T)
