"""The host-buffer drop-ins cut into more groups of chunks than they have lanes,
so that each lane's buffers, index and workspaces are used again by a later group
while the earlier one's output leaves.  The least size of a group is lowered for
these tests; how many groups a call is cut into is checked, so that they cannot
pass on another path.  Streams, sums and floats are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

EB, L = float(np.float32(2e-4)), 32
# n, T, groups with a least group of 2^19 elements
CASES = [(1 << 22, 16, 8), (24 * 174763 + 1, 24, 8), ((7 << 19) + 2, 7, 5), ((5 << 19) + 1, 5, 4), (72 * 43691, 72, 6),
         ((1 << 22) + 9, 18, 5)]


def groups(n, T):
    try:
        return Z.lib().zccl_gpu_dropin_groups(n, L, T)
    except OSError:
        pytest.skip("library not built")


def test_groups_of_a_call(monkeypatch):
    monkeypatch.delenv("ZCCL_GPU_TEST_LEAST_GROUP", raising=False)
    assert [groups(n, 16) for n in (1 << 22, (1 << 24) - 1, 1 << 24, 3 << 23, 1 << 25, 6 << 23, 1 << 27)] == [1, 1, 2, 3, 4, 6, 8]
    assert groups(1 << 24, 1) == 1 and groups((1 << 27) + 1, 3) == 3 and groups(3, 8) == 0
    assert groups((1 << 24) + 9, 16) == 1  # its last group of 8 chunks would not exceed the remainder
    monkeypatch.setenv("ZCCL_GPU_TEST_LEAST_GROUP", str(1 << 19))
    assert [groups(n, T) for n, T, _ in CASES] == [k for _, _, k in CASES]


@pytest.fixture
def small_groups(monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    monkeypatch.setenv("ZCCL_GPU_TEST_LEAST_GROUP", str(1 << 19))
    return torch


def wave(n, f):
    rng = np.random.default_rng(n)
    x = np.sin(np.arange(n, dtype=np.float32) * np.float32(f))
    x[: n // 2] += rng.normal(0, 0.01, n // 2).astype(np.float32)
    x[n // 3: n // 3 + n // 20] = 0
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("n,T,k", CASES)
@pytest.mark.parametrize("pinned", [False, True])
def test_more_groups_than_lanes(small_groups, port, n, T, k, pinned):
    torch = small_groups
    assert groups(n, T) == k
    x, y = wave(n, 1e-3), wave(n, 7e-4)
    sx, sy = port.compress(x, EB, L, T), port.compress(y, EB, L, T)
    dx, sxy = port.decompress(sx, n, EB, L, T).view(np.uint32), port.homadd(sx, sy, n, EB, L, T)
    cap = 4 * n + 8 * T + 4096

    def host(count, dtype):
        return torch.zeros(count, dtype=dtype, pin_memory=pinned).numpy()

    xh, yh, hs, acc, sep = host(n, torch.float32), host(n, torch.float32), *(host(cap, torch.uint8) for _ in range(3))
    Z.set_omp_threads(T)  # (torch sets its own count)
    for _ in range(3):  # buffers and indexes of the calls before are used again
        xh[:] = x
        hs[:] = sep[:] = 0
        assert Z.ZCCL_float_openmp_threadblock_arg(hs, xh, 0, EB, n, L) == len(sx)
        assert hs[: len(sx)].tobytes() == sx
        yh[:] = 0
        Z.ZCCL_float_decompress_openmp_threadblock_arg(yh, n, EB, L, hs)
        assert np.array_equal(yh.view(np.uint32), dx)
        acc[: len(sy)] = np.frombuffer(sy, np.uint8)
        total = Z.ZCCL_float_homomophic_add_openmp_threadblock(sep, 0, n, EB, L, hs, acc)
        assert total == len(sxy) and sep[:total].tobytes() == sxy
        total = Z.ZCCL_float_homomophic_add_openmp_threadblock(acc, 0, n, EB, L, hs, acc)
        assert total == len(sxy) and acc[:total].tobytes() == sxy


@pytest.mark.gpu
def test_bad_streams_in_any_group(small_groups, port):
    n, T = 1 << 22, 16
    assert groups(n, T) == 8
    good = port.compress(wave(n, 1e-3), EB, L, T)
    both = port.homadd(good, good, n, EB, L, T)
    floats = port.decompress(good, n, EB, L, T).view(np.uint32)
    hdr = np.frombuffer(good[: 8 * T], "<u8")
    Z.set_omp_threads(T)
    out = np.zeros(n, np.float32)

    def host(b):
        h = np.zeros(4 * n + 8 * T + 4096, np.uint8)
        h[: len(b)] = np.frombuffer(b, np.uint8)
        return h

    for chunk in (0, 6, 11, 15):  # the first group, groups of the first and second turn of the lanes, the last
        bad = host(good)
        bad[8 * T + int(hdr[chunk]) + 4:][:48] = 0xEE  # no width bytes
        with pytest.raises(Z.ZcclError):
            Z.ZCCL_float_decompress_openmp_threadblock_arg(out, n, EB, L, bad)
        for pair in ((bad, host(good)), (host(good), bad)):
            with pytest.raises(Z.ZcclError):
                Z.ZCCL_float_homomophic_add_openmp_threadblock(host(good), 0, n, EB, L, *pair)
        Z.ZCCL_float_decompress_openmp_threadblock_arg(out, n, EB, L, host(good))
        assert np.array_equal(out.view(np.uint32), floats)
        acc = host(good)
        total = Z.ZCCL_float_homomophic_add_openmp_threadblock(acc, 0, n, EB, L, host(good), acc)
        assert acc[:total].tobytes() == both
