"""The header walk on long runs of zero-width blocks, and on streams whose header
gives chunk offsets that do not increase: the walk's work then stays within its
scratch, which is sized for one stream of the worst size, and such a stream is
reported."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest


def test_windows_fit_the_scratch(tmp_path):
    """On the CPU, from the geometry the kernels and the scratch's layout
    share."""
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "walk_bounds"
    subprocess.run([cc, "-O2", "-I", os.path.join(here, "..", "zccl_gb300", "csrc"), "-o", str(exe),
                    os.path.join(here, "native", "walk_bounds.c")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    checked, over, refused = map(int, out.stdout.split())
    assert checked > 20_000 and over == 0 and refused == 0


@pytest.mark.gpu
@pytest.mark.parametrize("T", [2, 16, 72])
def test_alternating_offsets_are_reported(port, T):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import zccl_gb300 as Z
    n, L, eb = 1 << 20, 32, 1.0e-3
    x = np.cumsum(np.random.default_rng(T).normal(0, 0.01, n)).astype(np.float32)
    wire = port.compress(x, eb, L, T)
    codec = Z.Codec(n, L, T)
    body = len(wire) - 8 * T
    for far in (body - 8, body // 2, 100000 + 4 * n // T):
        bad = bytearray(wire)
        bad[: 8 * T] = np.array([far * (s & 1) for s in range(T)], "<u8").tobytes()
        codec.build_index(Z.DeviceStream.from_bytes(codec, bytes(bad)))
        with pytest.raises(Z.ZcclError):
            codec.check()
    s = Z.DeviceStream.from_bytes(codec, wire)
    y = codec.decompress(s, eb)
    codec.check()
    assert s.tobytes() == wire
    assert np.array_equal(y.cpu().numpy().view(np.uint32), port.decompress(wire, n, eb, L, T).view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("L", [8, 32, 36, 256])
@pytest.mark.parametrize("T", [1, 5])
def test_runs_of_zero_blocks(port, L, T):
    """Zero-width blocks, one byte each, in runs that end and begin at every
    place of a 16-byte line, alone and up to several windows long."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import zccl_gb300 as Z
    rng = np.random.default_rng(100 * L + T)
    runs = [1, 2, 14, 15, 16, 17, 31, 32, 33, 47, 48, 49, 200, 511, 512, 530, 2047, 2048, 2100, 6000]
    for seed in range(3):
        parts = []
        for r in rng.permutation(np.repeat(runs, 3)):
            parts += [np.zeros(int(r) * L), rng.normal(0, 10.0 ** rng.uniform(-3, 1), int(rng.integers(1, 8)) * L)]
        x = np.concatenate(parts).astype(np.float32)[: 1 << 21]
        if seed == 2:
            x[len(x) // 2:] = 0  # to the stream's end
        eb, n = 1.0e-3, x.size
        wire = port.compress(x, eb, L, T)
        want = port.decompress(wire, n, eb, L, T).view(np.uint32)
        codec = Z.Codec(n, L, T)
        for tail in (b"", b"\0" * 3000, b"\xff" * 100):
            s = Z.DeviceStream.from_bytes(codec, wire + tail)
            y = codec.decompress(s, eb)
            codec.check()
            assert s.tobytes() == wire
            assert np.array_equal(y.cpu().numpy().view(np.uint32), want)
