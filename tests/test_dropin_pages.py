"""The host-buffer drop-ins into output arrays in pages that nothing has touched:
the outputs are the oracle's, at any offset into a page, nothing behind them is
written, and an array that ends with its mapping is not reached past."""
from __future__ import annotations

import ctypes
import mmap

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu
EB, L, T = float(np.float32(2e-4)), 32, 8


class Fresh:
    """nbytes of fresh private memory, `gap` bytes from the mapping's end, behind
    which lies a page that may not be touched."""

    def __init__(self, nbytes, gap):
        libc = self.libc = ctypes.CDLL(None, use_errno=True)
        libc.mmap.restype = ctypes.c_void_p
        libc.mmap.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_long]
        libc.mprotect.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
        page = mmap.PAGESIZE
        room = -(-(nbytes + gap) // page) * page
        self.base, self.size = libc.mmap(None, room + page, 3, 0x22, -1, 0), room + page
        assert libc.mprotect(self.base + room, page, 0) == 0
        self.at = self.base + room - gap - nbytes
        self.bytes = np.frombuffer((ctypes.c_uint8 * (nbytes + gap)).from_address(self.at), np.uint8)


@pytest.mark.parametrize("gap", [0, 16, 4100])
@pytest.mark.parametrize("n", [70000, 1 << 20, (1 << 22) + 5])
@pytest.mark.parametrize("groups", [False, True])
def test_outputs_in_fresh_pages(port, monkeypatch, n, gap, groups):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if groups:
        monkeypatch.setenv("ZCCL_GPU_TEST_LEAST_GROUP", str(n // 5))
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal(0, 0.001, n)).astype(np.float32)
    wire = port.compress(x, EB, L, T)
    total = port.homadd(wire, wire, n, EB, L, T)
    floats = port.decompress(total, n, EB, L, T).view(np.uint32)
    src = np.zeros(4 * n + 8 * T + 4096, np.uint8)
    src[: len(wire)] = np.frombuffer(wire, np.uint8)
    both = np.zeros_like(src)
    both[: len(total)] = np.frombuffer(total, np.uint8)
    Z.set_omp_threads(T)
    assert (Z.lib().zccl_gpu_dropin_groups(n, L, T) > 1) == groups
    for _ in range(2):
        out = Fresh(len(wire), gap)
        assert Z.ZCCL_float_openmp_threadblock_arg(out.bytes, x, 0, EB, n, L) == len(wire)
        assert out.bytes[: len(wire)].tobytes() == wire and not out.bytes[len(wire):].any()
        out = Fresh(len(total), gap)
        assert Z.ZCCL_float_homomophic_add_openmp_threadblock(out.bytes, 0, n, EB, L, src, src) == len(total)
        assert out.bytes[: len(total)].tobytes() == total and not out.bytes[len(total):].any()
        y = Fresh(4 * n, gap)
        Z.ZCCL_float_decompress_openmp_threadblock_arg(y.bytes, n, EB, L, both)
        assert np.array_equal(y.bytes[: 4 * n].view(np.uint32), floats) and not y.bytes[4 * n:].any()
